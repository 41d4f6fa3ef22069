// Vertex-id hash join: HashJoin::build / HashJoin::probe
// (src/objects/operator/join.cpp:26-449) re-designed for sm_103a.
//
// Flat x Flat: an open-addressing table in HBM (64-bit keys, linear probing,
// load factor <= 1/2) is built over the smaller side; duplicate keys inside a
// warp are merged with __match_any_sync before one atomic per distinct key, so
// Zipf-skewed keys do not serialise on one slot.  Build rows are grouped by
// key (prefix sum over slot counts + scatter); the probe counts matches per
// probe row, a prefix sum places every probe row's output, and the emit pass
// assigns output rows to threads evenly (a thread binary-searches its probe
// row inside its block's range), so hot keys do not leave one thread writing
// millions of rows.
//
// Matrix operands are relations of (row value, column value) pairs with the
// column variable as key.  Count-only joins never materialise them:
// Flat x Mat sums multiplicity(key) * popcount(column) and Mat x Mat sums
// popcount(a column) * popcount(b column) per shared key, streaming each
// matrix once.  Materialising joins with a matrix operand expand its set
// bits to pairs (TableConvert(Flat)) and run the flat join.
#include <algorithm>
#include <cstring>
#include <mutex>

#include "dev_util.cuh"
#include "hash.cuh"
#include "vs_internal.cuh"

namespace vs {
namespace jn {

constexpr unsigned FULL = 0xffffffffu;
constexpr unsigned long long EMPTY = HT_EMPTY;
using Table = HashTable;

// Rows per vertex-id key, in an array indexed by the key (below, at k_key_max).
struct Direct {
  uint32_t *cnt;
  uint32_t bound;  // entries of the array
  uint32_t *top;   // largest build key
};

__device__ __forceinline__ bool direct_ok(const Direct &d) { return *d.top < d.bound; }

// The build side of a join that lists rows (below, at k_join_clear).
struct Build {
  Table t;               // keys (hash), rows per slot; off: first of the slot's rows, within its tile of 1,024 slots
  unsigned long long *tile_off;  // ... and the tile's
  uint32_t *row;         // by key: one plus a row that holds it
  uint32_t bound;        // keys the array has room for (0: none)
  uint32_t *ctl;         // [0] largest key, [1] some key has several rows, [2] [3] blocks of the scans that are done
  uint64_t n;            // rows
};
enum { J_HASH, J_ROWS, J_UNIQUE };

__device__ __forceinline__ int join_mode(const Build &b) {
  if (!b.bound || b.ctl[0] >= b.bound) return J_HASH;
  return b.ctl[1] ? J_ROWS : J_UNIQUE;
}

__device__ __forceinline__ unsigned long long load_key(const void *col, int type, uint64_t i) {
  return type == VS_T_I64 ? (unsigned long long)((const long long *)col)[i]
                          : (unsigned long long)((const uint32_t *)col)[i];
}

// Build: count rows per key.  Lanes holding the same key elect one leader
// that adds the group's size (skewed keys cost one atomic per warp).
template <class Slot>
__device__ __forceinline__ void build_rows(const Table &t, const void *keycol, int ktype, uint64_t lo, uint64_t n,
                                           uint32_t *slot_of, Slot find) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i0 = lo + (uint64_t)blockIdx.x * blockDim.x; i0 < n; i0 += stride) {
    const uint64_t i = i0 + threadIdx.x;
    const bool valid = i < n;
    const unsigned long long k = valid ? load_key(keycol, ktype, i) : EMPTY - 1;
    const unsigned active = __ballot_sync(FULL, valid);
    const unsigned peers = __match_any_sync(FULL, k) & active;
    if (valid) {
      const int leader = __ffs(peers) - 1;
      uint64_t slot = 0;
      if ((int)(threadIdx.x & 31) == leader) {
        slot = find(k, i);
        atomicAdd(&t.cnt[slot], (unsigned long long)__popc(peers));
      }
      slot = __shfl_sync(peers, slot, leader);
      if (slot_of) slot_of[i] = (uint32_t)slot;
    }
  }
}

__global__ void k_build(Table t, const void *keycol, int ktype, uint64_t n) {
  build_rows(t, keycol, ktype, 0, n, nullptr, [&](unsigned long long k, uint64_t) { return ht_insert(t, k); });
}

// Count-only build: each block first counts its rows' keys in a table of
// its own in shared memory and adds every key's block count to the global
// table once, so a hot key costs one global atomic per block instead of one
// per warp (a Zipf-skewed key column sends most warps to the same slot).
// Keys that find no shared slot within a few probes go to the global table
// directly.
constexpr int LOC_SLOTS = 4096;
__device__ __forceinline__ void build_count(const Table &t, const void *keycol, int ktype, uint64_t n,
                                            unsigned long long *s_key, uint32_t *s_cnt) {
  for (int i = threadIdx.x; i < LOC_SLOTS; i += blockDim.x) {
    s_key[i] = EMPTY;
    s_cnt[i] = 0;
  }
  __syncthreads();
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const unsigned long long k = load_key(keycol, ktype, i);
    bool done = false;
    if (k != EMPTY) {  // the all-ones key goes straight to its reserved global slot
      uint32_t h = (uint32_t)ht_hash(k) & (LOC_SLOTS - 1);
      for (int probe = 0; probe < 8 && !done; probe++) {
        unsigned long long old = s_key[h];
        if (old == EMPTY) old = atomicCAS(&s_key[h], EMPTY, k);
        if (old == EMPTY || old == k) {
          atomicAdd(&s_cnt[h], 1u);
          done = true;
        }
        h = (h + 1) & (LOC_SLOTS - 1);
      }
    }
    if (!done) {
      const uint64_t slot = ht_insert(t, k);
      atomicAdd(&t.cnt[slot], 1ull);
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < LOC_SLOTS; i += blockDim.x)
    if (s_cnt[i]) {
      const uint64_t slot = ht_insert(t, s_key[i]);
      atomicAdd(&t.cnt[slot], (unsigned long long)s_cnt[i]);
    }
}

__global__ void __launch_bounds__(256) k_build_count(Table t, const void *keycol, int ktype, uint64_t n) {
  __shared__ unsigned long long s_key[LOC_SLOTS];
  __shared__ uint32_t s_cnt[LOC_SLOTS];
  build_count(t, keycol, ktype, n, s_key, s_cnt);
}

// ---------------------------------------------------------------------------
// Vertex-id keys below a bound of a few times the build rows need no hash: an
// array indexed by the key holds each key's count, in L2 where the hash table of 10M
// keys is 537 MB of HBM.  The largest build key is found on the
// device and every kernel checks it against the bound, so the host waits for
// nothing; above the bound the count's kernels use the hash table instead.  Count of
// 10M x 10M Zipf-skewed keys below 10M: 432 -> 117 us, of which counting the build
// keys (shared-memory atomics) 71.
__global__ void __launch_bounds__(256) k_key_max(const uint32_t *__restrict__ keys, uint64_t n, uint32_t *ctl) {
  uint32_t m = 0;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x, i0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint4 *k4 = reinterpret_cast<const uint4 *>(keys);  // a column starts on an allocation
  for (uint64_t i = i0; i < n / 4; i += stride) {
    const uint4 k = __ldg(k4 + i);
    m = max(max(max(m, k.x), max(k.y, k.z)), k.w);
  }
  if (i0 < (n & 3)) m = max(m, keys[(n & ~3ull) + i0]);
  m = __reduce_max_sync(FULL, m);
  if ((threadIdx.x & 31) == 0) atomicMax(ctl, m);
}

// Clears the part of the array that the keys use, or the hash table that takes its
// place.
__global__ void __launch_bounds__(256) k_direct_clear(Direct d, Table t) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x, i0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (direct_ok(d)) {
    const uint32_t n4 = *d.top / 4 + 1;  // the bound is a multiple of four
    for (uint64_t i = i0; i < n4; i += stride) reinterpret_cast<uint4 *>(d.cnt)[i] = make_uint4(0, 0, 0, 0);
  } else {
    for (uint64_t i = i0; i <= t.cap; i += stride) {
      t.keys[i] = EMPTY;
      t.cnt[i] = 0;
    }
  }
}

// Counts per key.  As in k_build_count a block first counts in a table of its own
// in shared memory (Zipf-skewed columns send an eighth of the rows to one key), with
// one probe: a key that finds the slot taken adds to the array in L2.
constexpr int DIRECT_SLOTS = LOC_SLOTS;
__global__ void __launch_bounds__(512) k_direct_count(Direct d, Table t, const uint32_t *__restrict__ keys, uint64_t n) {
  __shared__ unsigned long long s_wide[LOC_SLOTS];
  __shared__ uint32_t s_cnt[LOC_SLOTS];
  if (!direct_ok(d)) {
    build_count(t, keys, VS_T_VID, n, s_wide, s_cnt);
    return;
  }
  uint32_t *s_key = reinterpret_cast<uint32_t *>(s_wide);
  for (int i = threadIdx.x; i < DIRECT_SLOTS; i += blockDim.x) {
    s_key[i] = 0xffffffffu;  // not a key below the bound
    s_cnt[i] = 0;
  }
  __syncthreads();
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x, i0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  auto add = [&](uint32_t k) {
    const uint32_t h = (k * 2654435761u) >> 20;  // 12 bits
    uint32_t old = s_key[h];
    if (old == 0xffffffffu) old = atomicCAS(&s_key[h], 0xffffffffu, k);
    if (old == 0xffffffffu || old == k)
      atomicAdd(&s_cnt[h], 1u);
    else
      atomicAdd(&d.cnt[k], 1u);
  };
  const uint4 *k4 = reinterpret_cast<const uint4 *>(keys);
  for (uint64_t i = i0; i < n / 4; i += stride) {
    const uint4 k = __ldg(k4 + i);
    add(k.x);
    add(k.y);
    add(k.z);
    add(k.w);
  }
  if (i0 < (n & 3)) add(keys[(n & ~3ull) + i0]);
  __syncthreads();
  for (int i = threadIdx.x; i < DIRECT_SLOTS; i += blockDim.x)
    if (s_cnt[i]) atomicAdd(&d.cnt[s_key[i]], s_cnt[i]);
}

// Sum of the counts of the probe keys.
__global__ void __launch_bounds__(256) k_direct_probe(Direct d, Table t, const uint32_t *__restrict__ keys,
                                                      uint64_t n, unsigned long long *total) {
  const uint32_t top = *d.top;
  unsigned long long s = 0;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x, i0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (!direct_ok(d)) {
    for (uint64_t i = i0; i < n; i += stride) {
      const uint64_t slot = ht_find(t, keys[i]);
      if (slot != ~0ull) s += t.cnt[slot];
    }
    block_add(s, total);
    return;
  }
  const uint4 *k4 = reinterpret_cast<const uint4 *>(keys);
  for (uint64_t i = i0; i < n / 4; i += stride) {
    const uint4 k = __ldg(k4 + i);
    const uint32_t a = k.x <= top ? __ldg(d.cnt + k.x) : 0u, b = k.y <= top ? __ldg(d.cnt + k.y) : 0u;
    const uint32_t c = k.z <= top ? __ldg(d.cnt + k.z) : 0u, e = k.w <= top ? __ldg(d.cnt + k.w) : 0u;
    s += (unsigned long long)a + b + c + e;
  }
  if (i0 < (n & 3)) {
    const uint32_t k = keys[(n & ~3ull) + i0];
    if (k <= top) s += d.cnt[k];
  }
  block_add(s, total);
}

// Joins that list rows.  Vertex-id keys below a bound get their slot from an array
// indexed by the key that holds (one plus) a row with it: the row itself where every key
// has one (a property table: UNIQUE), else the row's number is the key's slot (ROWS);
// other keys get it from the hash table.  Which of the three it is the device finds on
// the way, and kernels that the mode has no use for return at once, so that the host
// waits once, for the number of rows: told first whether the keys are unique, a join
// of repeated keys waited some 40 us longer.  4M probe rows against 1M rows of five
// columns in all: unique keys 376 (hash table) -> 173 us, repeated ones 417 -> 400; 4,000
// against 1,000 rows of repeated keys 125 -> 98.
__global__ void __launch_bounds__(256) k_join_clear(Build b, int counts) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x, i0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (join_mode(b) == J_HASH) {
    for (uint64_t i = i0; i <= b.t.cap; i += stride) {
      b.t.keys[i] = EMPTY;
      b.t.cnt[i] = 0;
    }
  } else {
    const uint32_t n4 = b.ctl[0] / 4 + 1;  // the bound is a multiple of four
    for (uint64_t i = i0; i < n4; i += stride) reinterpret_cast<uint4 *>(b.row)[i] = make_uint4(0, 0, 0, 0);
    if (counts)
      for (uint64_t i = i0; i < b.n; i += stride) b.t.cnt[i] = 0;
  }
}

// Build rows [i_lo, i_hi) into the array, until a key is met again, or into the hash
// table.  The first rows come alone, with few blocks: in most tables with repeated keys one
// is met among them, and the atomics and stores of a full grid that meets one at the same
// time took 134 us for 1M rows.
__global__ void __launch_bounds__(256) k_join_build(Build b, const void *keycol, int ktype, uint32_t *slot_of, uint64_t i_lo,
                                                    uint64_t i_hi) {
  if (!b.bound || b.ctl[0] >= b.bound) {
    build_rows(b.t, keycol, ktype, i_lo, i_hi, slot_of, [&](unsigned long long k, uint64_t) { return ht_insert(b.t, k); });
    return;
  }
  const uint32_t *keys = (const uint32_t *)keycol;
  const unsigned lane = threadIdx.x & 31;
  for (uint64_t i0 = i_lo + (uint64_t)blockIdx.x * blockDim.x; i0 < i_hi; i0 += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t i = i0 + threadIdx.x;
    const bool known = __shfl_sync(FULL, __ldcg(b.ctl + 1), 0);
    if (known) return;
    const uint32_t k = i < i_hi ? __ldg(keys + i) : 0u;
    // a key twice in the warp needs no atomic (hot keys would queue at one address)
    const unsigned peers = __match_any_sync(FULL, i < i_hi ? (unsigned long long)k : EMPTY - lane);
    bool again = i < i_hi && (peers & lanemask_lt());
    if (!__any_sync(FULL, again) && i < i_hi) again = atomicExch(&b.row[k], (uint32_t)i + 1) != 0;
    if (__any_sync(FULL, again)) {
      if (lane == 0 && !__ldcg(b.ctl + 1)) b.ctl[1] = 1;
      return;
    }
  }
}

// Repeated keys: the array completed, and rows per slot.
__global__ void __launch_bounds__(256) k_join_count(Build b, const uint32_t *__restrict__ keys, uint32_t *slot_of) {
  if (join_mode(b) != J_ROWS) return;
  build_rows(b.t, keys, VS_T_VID, 0, b.n, slot_of, [&](unsigned long long k, uint64_t i) {
    uint32_t r = __ldcg(b.row + k);
    if (!r) {
      r = atomicCAS(&b.row[k], 0u, (uint32_t)i + 1);
      if (!r) r = (uint32_t)i + 1;
    }
    return (uint64_t)(r - 1);
  });
}

// Exclusive prefix in one launch: out within tiles of 1,024, and by the block that
// finishes last the tiles' starts.  n_hash elements in HASH mode, n_rows in ROWS mode;
// element n gets the total.
__global__ void __launch_bounds__(256) k_join_scan(Build b, const unsigned long long *__restrict__ in,
                                                   unsigned long long *__restrict__ out, unsigned long long *tile_off,
                                                   uint64_t n_hash, uint64_t n_rows, uint32_t *done) {
  const int mode = join_mode(b);
  if (mode == J_UNIQUE) return;
  const uint64_t n = mode == J_HASH ? n_hash : n_rows, tiles = n / 1024 + 1;  // element n has a tile too
  if (blockIdx.x >= tiles) return;
  __shared__ unsigned long long wt[8];
  __shared__ bool s_last;
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  unsigned long long v[4] = {0, 0, 0, 0};
  auto scan4 = [&]() {  // v becomes the exclusive prefix over the block's 1,024 values; returns their sum
    const unsigned long long run = v[0] + v[1] + v[2] + v[3];
    unsigned long long incl = run;
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long y = __shfl_up_sync(FULL, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) wt[w] = incl;
    __syncthreads();
    unsigned long long pre = 0, sum = 0;
    for (int k = 0; k < 8; k++) {
      if (k < w) pre += wt[k];
      sum += wt[k];
    }
    pre += incl - run;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const unsigned long long x = v[k];
      v[k] = pre;
      pre += x;
    }
    __syncthreads();
    return sum;
  };
  for (uint64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const uint64_t base = tile * 1024 + (uint64_t)t * 4;
#pragma unroll
    for (int k = 0; k < 4; k++) v[k] = base + k < n ? in[base + k] : 0ull;
    const unsigned long long sum = scan4();
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (base + k <= n) out[base + k] = v[k];
    if (t == 0) tile_off[tile] = sum;
  }
  __threadfence();
  __syncthreads();
  const uint64_t blocks = tiles < gridDim.x ? tiles : gridDim.x;
  if (t == 0) s_last = atomicAdd(done, 1u) == blocks - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  unsigned long long carry = 0;
  for (uint64_t b0 = 0; b0 < tiles; b0 += 1024) {
    const uint64_t base = b0 + (uint64_t)t * 4;
#pragma unroll
    for (int k = 0; k < 4; k++) v[k] = base + k < tiles ? __ldcg(tile_off + base + k) : 0ull;
    const unsigned long long sum = scan4();
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (base + k < tiles) tile_off[base + k] = carry + v[k];
    carry += sum;
  }
}

__device__ __forceinline__ unsigned long long start_of(const unsigned long long *__restrict__ off,
                                                       const unsigned long long *__restrict__ tile_off, uint64_t i) {
  return off[i] + tile_off[i >> 10];
}

// Build rows by slot (the counts go down to zero); one lane takes the places of a
// warp's rows of one slot (300K rows, 38% of one key: 106 -> 32 us).
__global__ void __launch_bounds__(256) k_join_scatter(Build b, const uint32_t *__restrict__ slot_of,
                                                      uint32_t *__restrict__ rows_by_key) {
  if (join_mode(b) == J_UNIQUE) return;
  const unsigned lane = threadIdx.x & 31;
  for (uint64_t i0 = (uint64_t)blockIdx.x * blockDim.x; i0 < b.n; i0 += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t i = i0 + threadIdx.x;
    const uint32_t s = i < b.n ? slot_of[i] : 0u;
    const unsigned peers = __match_any_sync(FULL, i < b.n ? (unsigned long long)s : EMPTY - lane);
    const int leader = __ffs(peers) - 1;
    unsigned long long at = 0;
    if (i < b.n && (int)lane == leader)
      at = start_of(b.t.off, b.tile_off, s) + atomicAdd(&b.t.cnt[s], 0ull - __popc(peers)) - __popc(peers);
    at = __shfl_sync(FULL, at, leader);
    if (i < b.n) rows_by_key[at + __popc(peers & lanemask_lt())] = (uint32_t)i;
  }
}

// Probe.  UNIQUE: matching rows per tile of FK_ROWS (sums[tile]); else matches per row
// and the row's slot.  All of them in *total.
constexpr int FK_ROWS = 1024;
__global__ void __launch_bounds__(256) k_join_probe(Build b, const void *keycol, int ktype, uint64_t n,
                                                    unsigned long long *__restrict__ sums,
                                                    unsigned long long *__restrict__ pcnt, uint32_t *__restrict__ pslot,
                                                    unsigned long long *total, int unique_only) {
  const int mode = join_mode(b);
  if (unique_only && mode != J_UNIQUE) return;
  const uint32_t *keys = (const uint32_t *)keycol;
  const uint32_t top = b.ctl[0];
  unsigned long long all = 0;
  if (mode != J_UNIQUE) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
      uint64_t slot;
      if (mode == J_HASH) {
        slot = ht_find(b.t, load_key(keycol, ktype, i));
      } else {
        const uint32_t k = __ldg(keys + i);
        slot = k <= top ? (uint64_t)__ldg(b.row + k) - 1 : ~0ull;  // 0: no row
      }
      unsigned long long c = 0;
      if (slot != ~0ull) c = start_of(b.t.off, b.tile_off, slot + 1) - start_of(b.t.off, b.tile_off, slot);
      all += c;
      pcnt[i] = c;
      pslot[i] = (uint32_t)(slot == ~0ull ? 0 : slot);
    }
    block_add(all, total);
    return;
  }
  __shared__ uint32_t part[8];
  for (uint64_t tile = blockIdx.x; tile * FK_ROWS < n; tile += gridDim.x) {
    uint32_t c = 0;
#pragma unroll
    for (int k = 0; k < FK_ROWS / 256; k++) {
      const uint64_t i = tile * FK_ROWS + k * 256 + threadIdx.x;
      const uint32_t x = i < n ? __ldg(keys + i) : 0xffffffffu;
      c += x <= top && __ldg(b.row + x);
    }
    c = __reduce_add_sync(FULL, c);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
      uint32_t t = 0;
      for (int w = 0; w < 8; w++) t += part[w];
      sums[tile] = t;
      all += t;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0 && all) atomicAdd(total, all);
}

// Build over matrix columns: key = col_map[c] (or c) -> first column index.
__global__ void k_build_cols(Table t, const uint32_t *col_map, uint32_t cols) {
  for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < cols; c += gridDim.x * blockDim.x) {
    const unsigned long long k = col_map ? col_map[c] : c;
    const uint64_t s = ht_insert(t, k);
    atomicMin(&t.val[s], c);
    atomicAdd(&t.cnt[s], 1ull);
  }
}

// Probe: sum of the counts of the probe keys.
__global__ void k_probe(Table t, const void *keycol, int ktype, uint64_t n, unsigned long long *total) {
  unsigned long long s = 0;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t slot = ht_find(t, load_key(keycol, ktype, i));
    if (slot != ~0ull) s += t.cnt[slot];
  }
  block_add(s, total);
}

// Flat x Mat count: sum over matrix columns of multiplicity(key) * popcount.
__global__ void k_count_mat(Table t, const uint64_t *__restrict__ w, uint32_t cols, uint32_t wpc,
                            const uint32_t *col_map, unsigned long long *total) {
  const int lane = threadIdx.x & 31;
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  unsigned long long s = 0;
  for (uint32_t c = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); c < cols; c += warps) {
    unsigned long long m = 0;
    if (lane == 0) {
      const uint64_t slot = ht_find(t, col_map ? col_map[c] : c);
      m = slot == ~0ull ? 0ull : t.cnt[slot];
    }
    m = __shfl_sync(FULL, m, 0);
    if (!m) continue;
    unsigned long long pc = 0;
    for (uint32_t q = lane; q < wpc; q += 32) pc += __popcll(w[(size_t)c * wpc + q]);
    pc = warp_sum(pc);
    if (lane == 0) s += m * pc;
  }
  block_add(s, total);
}

// Mat x Mat count: for every column of b, the column of a with the same key.
__global__ void k_count_mat_mat(Table ta, const uint64_t *__restrict__ wa, uint32_t cols_a,
                                uint32_t wpc_a, const uint64_t *__restrict__ wb, uint32_t cols_b,
                                uint32_t wpc_b, const uint32_t *col_map_b, int direct,
                                unsigned long long *total) {
  const int lane = threadIdx.x & 31;
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  unsigned long long s = 0;
  for (uint32_t c = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); c < cols_b; c += warps) {
    uint32_t ca = 0xffffffffu;
    if (direct) {
      ca = c < cols_a ? c : 0xffffffffu;
    } else if (lane == 0) {
      const uint64_t slot = ht_find(ta, col_map_b ? col_map_b[c] : c);
      ca = slot == ~0ull ? 0xffffffffu : ta.val[slot];
    }
    ca = __shfl_sync(FULL, ca, 0);
    if (ca == 0xffffffffu) continue;
    unsigned long long pa = 0, pb = 0;
    for (uint32_t q = lane; q < wpc_a; q += 32) pa += __popcll(wa[(size_t)ca * wpc_a + q]);
    for (uint32_t q = lane; q < wpc_b; q += 32) pb += __popcll(wb[(size_t)c * wpc_b + q]);
    pa = warp_sum(pa);
    pb = warp_sum(pb);
    if (lane == 0) s += pa * pb;
  }
  block_add(s, total);
}

// Mat x Mat count when neither operand has a column map (key = column index):
// a warp takes 32 columns, keeps those that may be non-zero in both, and
// popcounts each pair of columns with 16-byte loads and one warp reduction.
__global__ void __launch_bounds__(256) k_count_direct(const uint4 *__restrict__ wa, uint32_t qa,
                                                      const uint4 *__restrict__ wb, uint32_t qb, uint32_t cols,
                                                      const uint32_t *__restrict__ nza,
                                                      const uint32_t *__restrict__ nzb,
                                                      unsigned long long *total) {
  const int lane = threadIdx.x & 31;
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  unsigned long long s = 0;
  for (uint32_t c0 = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * 32; c0 < cols; c0 += warps * 32) {
    const uint32_t cl = c0 + lane;
    unsigned m = __ballot_sync(FULL, cl < cols && (!nza || nza[cl]) && (!nzb || nzb[cl]));
    while (m) {
      const uint32_t c = c0 + __ffs(m) - 1;
      m &= m - 1;
      unsigned pa = 0, pb = 0;
      for (uint32_t q = lane; q < qa; q += 32) {
        const uint4 x = __ldg(wa + (size_t)c * qa + q);
        pa += __popc(x.x) + __popc(x.y) + __popc(x.z) + __popc(x.w);
      }
      for (uint32_t q = lane; q < qb; q += 32) {
        const uint4 x = __ldg(wb + (size_t)c * qb + q);
        pb += __popc(x.x) + __popc(x.y) + __popc(x.z) + __popc(x.w);
      }
      pa = __reduce_add_sync(FULL, pa);
      pb = __reduce_add_sync(FULL, pb);
      s += (unsigned long long)pa * pb;
    }
  }
  if (lane != 0) s = 0;
  block_add(s, total);
}

struct OutCol {
  void *dst;
  const void *src;
  int type;
  int side;  // 0 = probe row, 1 = build row
};

struct EmitArgs {
  OutCol col[16];
  int ncols;
  const unsigned long long *poff, *ptile;  // first output row of every probe row, within its tile and the tile's
  const uint32_t *pslot;
  const uint32_t *rows_by_key;
  Build b;
  uint64_t n_probe, out_rows;
};

// Output rows [blk*R, blk*R + R) of every block; thread -> probe row by a
// binary search of the rows' starts inside the block's probe range.
constexpr int EMIT_ROWS = 2048;

__global__ void __launch_bounds__(256) k_emit(EmitArgs a) {
  __shared__ uint64_t p_lo, p_hi;
  __shared__ unsigned long long s_start[EMIT_ROWS];
  const uint64_t o0 = (uint64_t)blockIdx.x * EMIT_ROWS;
  if (o0 >= a.out_rows) return;
  const uint64_t o1 = min(o0 + EMIT_ROWS, a.out_rows);
  if (threadIdx.x == 0) {
    // largest p that starts at or before o0, and at or before o1 - 1
    uint64_t lo = 0, hi = a.n_probe;
    while (hi - lo > 1) {
      uint64_t mid = (lo + hi) / 2;
      if (start_of(a.poff, a.ptile, mid) <= o0) lo = mid; else hi = mid;
    }
    p_lo = lo;
    uint64_t lo2 = lo, hi2 = a.n_probe;
    while (hi2 - lo2 > 1) {
      uint64_t mid = (lo2 + hi2) / 2;
      if (start_of(a.poff, a.ptile, mid) <= o1 - 1) lo2 = mid; else hi2 = mid;
    }
    p_hi = lo2;
  }
  __syncthreads();
  const bool held = p_hi - p_lo < EMIT_ROWS;  // the range's starts fit
  if (held)
    for (uint64_t p = p_lo + threadIdx.x; p <= p_hi; p += blockDim.x) s_start[p - p_lo] = start_of(a.poff, a.ptile, p);
  __syncthreads();
  for (uint64_t o = o0 + threadIdx.x; o < o1; o += blockDim.x) {
    uint64_t lo = p_lo, hi = p_hi + 1;
    while (hi - lo > 1) {
      uint64_t mid = (lo + hi) / 2;
      if ((held ? s_start[mid - p_lo] : start_of(a.poff, a.ptile, mid)) <= o) lo = mid; else hi = mid;
    }
    const uint64_t p = lo;
    const uint64_t j = o - (held ? s_start[p - p_lo] : start_of(a.poff, a.ptile, p));
    const uint32_t s = a.pslot[p];
    const uint64_t b = a.rows_by_key[start_of(a.b.t.off, a.b.tile_off, s) + j];
    for (int c = 0; c < a.ncols; c++) {
      const OutCol &oc = a.col[c];
      const uint64_t r = oc.side ? b : p;
      if (oc.type == VS_T_I64)
        ((long long *)oc.dst)[o] = ((const long long *)oc.src)[r];
      else
        ((uint32_t *)oc.dst)[o] = ((const uint32_t *)oc.src)[r];
    }
  }
}

// Output rows of the matching probe rows of each tile, in probe order: one build
// row each, so a row's place is the tile's offset plus its rank among the tile's
// matches and no per-row counts, offsets or slots go through memory.  Bound by random
// sectors, one for the row and one per build column: the row sits in the key's word
// itself (a count and a row array: 54 -> 44 us for 4M rows of 20 bytes).
__global__ void __launch_bounds__(256) k_fk_emit(EmitArgs a, const uint32_t *__restrict__ keys,
                                                 const unsigned long long *__restrict__ tile_off) {
  const uint32_t top = a.b.ctl[0];
  __shared__ uint32_t part[FK_ROWS / 32];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (uint64_t b = blockIdx.x; b * FK_ROWS < a.n_probe; b += gridDim.x) {
    const unsigned long long o0 = tile_off[b];
    if (o0 >= a.out_rows) return;  // later tiles lie past the caller's bound too
    uint32_t row[FK_ROWS / 256];
    unsigned hit[FK_ROWS / 256];
#pragma unroll
    for (int k = 0; k < FK_ROWS / 256; k++) {
      const uint64_t i = b * FK_ROWS + k * 256 + threadIdx.x;
      row[k] = i < a.n_probe ? __ldg(keys + i) : 0xffffffffu;
    }
#pragma unroll
    for (int k = 0; k < FK_ROWS / 256; k++) row[k] = row[k] <= top ? __ldg(a.b.row + row[k]) : 0u;  // one plus the row
#pragma unroll
    for (int k = 0; k < FK_ROWS / 256; k++) {
      hit[k] = __ballot_sync(FULL, row[k] != 0);
      if (lane == 0) part[k * 8 + warp] = __popc(hit[k]);
    }
    __syncthreads();
    if (warp == 0) {  // FK_ROWS / 32 == 32: a lane per warp-row
      const uint32_t x = part[lane];
      uint32_t incl = x;
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(FULL, incl, o);
        if (lane >= (uint32_t)o) incl += y;
      }
      part[lane] = incl - x;
    }
    __syncthreads();
    for (int c = 0; c < a.ncols; c++) {
      const OutCol oc = a.col[c];
#pragma unroll
      for (int k = 0; k < FK_ROWS / 256; k++) {
        const uint64_t i = b * FK_ROWS + k * 256 + threadIdx.x;
        const unsigned long long o = o0 + part[k * 8 + warp] + __popc(hit[k] & lanemask_lt());
        if (!(hit[k] >> lane & 1u) || o >= a.out_rows) continue;
        const uint64_t r = oc.side ? (uint64_t)row[k] - 1 : i;
        if (oc.type == VS_T_I64)
          ((long long *)oc.dst)[o] = __ldg((const long long *)oc.src + r);
        else
          ((uint32_t *)oc.dst)[o] = __ldg((const uint32_t *)oc.src + r);
      }
    }
    __syncthreads();
  }
}

// One allocation for the arrays of a call: an allocation and its release cost the host
// about 1.5 us, a small join has ten.
struct Scratch {
  cudaStream_t st;
  char *base = nullptr;
  size_t bytes = 0;
  explicit Scratch(cudaStream_t s) : st(s) {}
  template <typename T> size_t add(size_t n) {  // offset of n elements
    const size_t at = bytes;
    bytes += (sizeof(T) * (n ? n : 1) + 255) / 256 * 256;
    return at;
  }
  int alloc() { return dalloc_n(&base, bytes, st); }
  template <typename T> T *at(size_t off) const { return reinterpret_cast<T *>(base + off); }
  void release() {  // the layout stays
    dfree(base, st);
    base = nullptr;
  }
  ~Scratch() { release(); }
};

// A hash table's arrays within a scratch, and `extra` elements of 8 bytes zeroed with its
// counters.
struct TablePart {
  size_t keys = 0, cnt = 0, zeroed = 0, end = 0, val = 0;
  bool with_val = false;
  uint64_t cap = 0;
  void add(Scratch &sc, uint64_t n_keys, bool val_, size_t extra) {
    cap = ht_capacity(std::max<uint64_t>(n_keys, 1));
    with_val = val_;
    keys = sc.add<uint64_t>(cap + 1);
    cnt = sc.add<uint64_t>(cap + 1);
    zeroed = extra ? sc.add<uint64_t>(extra) : sc.bytes;
    end = sc.bytes;
    val = val_ ? sc.add<uint32_t>(cap + 1) : 0;
  }
  Table table(const Scratch &sc) const {
    Table t{};
    t.cap = cap;
    t.keys = sc.at<unsigned long long>(keys);
    t.cnt = sc.at<unsigned long long>(cnt);
    if (with_val) t.val = sc.at<uint32_t>(val);
    return t;
  }
  int clear(const Scratch &sc) const {
    VS_CK(cudaMemsetAsync(sc.base + keys, 0xff, 8 * (cap + 1), sc.st));
    VS_CK(cudaMemsetAsync(sc.base + cnt, 0, end - cnt, sc.st));
    if (with_val) VS_CK(cudaMemsetAsync(sc.base + val, 0xff, 4 * (cap + 1), sc.st));
    return VS_OK;
  }
};

int grid_for(uint64_t n, int per_block = 256) {
  return (int)std::max<uint64_t>(1, std::min<uint64_t>((n + per_block - 1) / per_block,
                                                       (uint64_t)sm_count() * 16));
}

int read_total(unsigned long long *d, uint64_t *h, cudaStream_t st) {
  unsigned long long x = 0;
  VS_CK(cudaMemcpyAsync(&x, d, sizeof(x), cudaMemcpyDeviceToHost, st));
  VS_CK(cudaStreamSynchronize(st));
  *h = x;
  return VS_OK;
}

// A flat operand: columns + key column.
struct FlatSide {
  const vs_flat *f;
  uint32_t key;
};

// Key bound up to which an array indexed by the key is used: 4 bytes an entry where a
// hash table takes 32 to 64 a row.  Below 4M entries (16 MB, cleared in 5 us, in L2) it
// wins whatever the rows.  Above, counts take it up to 4 entries a row, joins that list
// rows up to 12 (1M rows, keys below 12M: unique 366 -> 184 us, repeated 362 -> 361;
// keys above, 40M: 6% slower than without asking for the largest key).
uint32_t direct_bound(uint64_t n_build, uint64_t per_row) {
  return n_build > (1ull << 27) ? 0u : (uint32_t)std::max<uint64_t>(1u << 22, per_row * n_build / 4 * 4);
}

// Result schema: a's columns, then b's non-key columns.
int join_columns(FlatSide a, FlatSide b, bool build_a, int32_t *types, EmitArgs *ea) {
  int nc = 0;
  for (uint32_t i = 0; i < a.f->ncols; i++) {
    types[nc] = a.f->types[i];
    ea->col[nc].src = a.f->cols[i];
    ea->col[nc].type = a.f->types[i];
    ea->col[nc].side = build_a ? 1 : 0;
    nc++;
  }
  for (uint32_t i = 0; i < b.f->ncols; i++) {
    if (i == b.key) continue;
    if (nc >= 16) return fail(VS_ERR_UNSUPPORTED, "join result wider than 16 columns");
    types[nc] = b.f->types[i];
    ea->col[nc].src = b.f->cols[i];
    ea->col[nc].type = b.f->types[i];
    ea->col[nc].side = build_a ? 0 : 1;
    nc++;
  }
  ea->ncols = nc;
  return VS_OK;
}

// Count of a flat join: of vertex-id keys through the array indexed by the key, or the
// hash table in its place (chosen on the device), of others through the hash table.
int count_flat_flat(FlatSide bd, FlatSide pr, uint64_t *count, cudaStream_t st) {
  const uint64_t nb = bd.f->nrows, np = pr.f->nrows;
  const uint32_t *bkeys = (const uint32_t *)bd.f->cols[bd.key], *pkeys = (const uint32_t *)pr.f->cols[pr.key];
  const uint32_t bound = bd.f->types[bd.key] == VS_T_VID && nb && np ? direct_bound(nb, 4) : 0u;
  Scratch sc{st};
  TablePart tp;
  if (bound) {
    tp.add(sc, nb, false, 0);
    const size_t o_ctl = sc.add<uint64_t>(2), o_cnt = sc.add<uint32_t>(bound);
    const int rc = sc.alloc();
    if (rc != VS_OK && rc != VS_ERR_OOM) return rc;
    if (rc == VS_OK) {
      const Table t = tp.table(sc);
      unsigned long long *d_total = sc.at<unsigned long long>(o_ctl);
      const Direct d{sc.at<uint32_t>(o_cnt), bound, reinterpret_cast<uint32_t *>(d_total + 1)};
      VS_CK(cudaMemsetAsync(d_total, 0, 16, st));
      { k_key_max<<<std::min(grid_for((nb + 3) / 4), 4 * sm_count()), 256, 0, st>>>(bkeys, nb, d.top); vs::note_launch(); }
      { k_direct_clear<<<std::min(grid_for((bound + 3) / 4), 8 * sm_count()), 256, 0, st>>>(d, t); vs::note_launch(); }
      { k_direct_count<<<std::min(grid_for(nb, 512), 2 * sm_count()), 512, 0, st>>>(d, t, bkeys, nb); vs::note_launch(); }
      { k_direct_probe<<<grid_for(np), 256, 0, st>>>(d, t, pkeys, np, d_total); vs::note_launch(); }
      VS_CK(cudaGetLastError());
      return read_total(d_total, count, st);
    }
    sc.bytes = 0;  // no room for both
  }
  tp.add(sc, nb, false, 1);
  VS_TRY(sc.alloc());
  VS_TRY(tp.clear(sc));
  const Table t = tp.table(sc);
  unsigned long long *d_total = sc.at<unsigned long long>(tp.zeroed);
  if (nb)
    { k_build_count<<<std::min(grid_for(nb), 4 * sm_count()), 256, 0, st>>>(t, bkeys, bd.f->types[bd.key], nb); vs::note_launch(); }
  if (np)
    { k_probe<<<grid_for(np), 256, 0, st>>>(t, pkeys, pr.f->types[pr.key], np, d_total); vs::note_launch(); }
  VS_CK(cudaGetLastError());
  return read_total(d_total, count, st);
}

// Build rows from which a join that lists rows asks whether the keys are unique before it
// goes on (at `early`).
constexpr uint64_t ASK_ROWS = 512 << 10;

// Flat x Flat join.  a = deps[0], b = deps[1]; result = a cols + b non-key cols.
int join_flat_flat(FlatSide a, FlatSide b, bool only_count, uint64_t max_rows, vs_flat **out,
                   uint64_t *count, cudaStream_t st) {
  if (a.f->types[a.key] != b.f->types[b.key])
    return fail(VS_ERR_ARG, "join key types differ (%d vs %d)", a.f->types[a.key], b.f->types[b.key]);
  // GPU build side: the smaller table (the reference builds on the larger,
  // join.cpp:39-43; the side only changes the output order)
  const bool build_a = a.f->nrows < b.f->nrows;
  const FlatSide &bd = build_a ? a : b, &pr = build_a ? b : a;
  if (only_count) return count_flat_flat(bd, pr, count, st);
  const uint64_t nb = bd.f->nrows, np = pr.f->nrows;
  const int ktype = bd.f->types[bd.key];
  const void *bkeys = bd.f->cols[bd.key], *pkeys = pr.f->cols[pr.key];
  Build d{};
  d.n = nb;
  d.bound = ktype == VS_T_VID && nb && np ? direct_bound(nb, 12) : 0u;
  const uint64_t tiles = (np + FK_ROWS - 1) / FK_ROWS;
  Scratch sc{st};
  TablePart tp;
  size_t o_ctl, o_off, o_toff, o_slot, o_rows, o_pcnt, o_poff, o_ptile, o_pslot, o_row;
  for (;;) {
    sc.bytes = 0;
    tp.add(sc, nb, false, 0);
    o_ctl = sc.add<uint64_t>(3);  // total, then the control words
    o_off = sc.add<uint64_t>(tp.cap + 2);
    o_toff = sc.add<uint64_t>((tp.cap + 1) / 1024 + 1);
    o_slot = sc.add<uint32_t>(nb);
    o_rows = sc.add<uint32_t>(nb);
    o_pcnt = sc.add<uint64_t>(np);
    o_poff = sc.add<uint64_t>(np + 1);
    o_ptile = sc.add<uint64_t>(np / 1024 + 1);
    o_pslot = sc.add<uint32_t>(np);
    o_row = sc.add<uint32_t>(d.bound);
    const int rc = sc.alloc();
    if (rc == VS_OK) break;
    if (rc != VS_ERR_OOM || !d.bound) return rc;
    d.bound = 0;  // without the array
  }
  d.t = tp.table(sc);
  d.t.off = sc.at<unsigned long long>(o_off);
  d.tile_off = sc.at<unsigned long long>(o_toff);
  d.row = sc.at<uint32_t>(o_row);
  unsigned long long *d_total = sc.at<unsigned long long>(o_ctl), *pcnt = sc.at<unsigned long long>(o_pcnt),
                     *poff = sc.at<unsigned long long>(o_poff), *ptile = sc.at<unsigned long long>(o_ptile);
  d.ctl = reinterpret_cast<uint32_t *>(d_total + 1);
  uint32_t *slot_of = sc.at<uint32_t>(o_slot), *rows_by_key = sc.at<uint32_t>(o_rows), *pslot = sc.at<uint32_t>(o_pslot);
  unsigned long long *sums = pcnt, *offs = poff;  // UNIQUE: by tile
  const int cap_grid = 8 * sm_count();
  // a wait more costs a join of repeated keys some 10 us; the kernels that a join of
  // unique keys does not need cost it as much
  const bool early = d.bound && nb >= ASK_ROWS;
  VS_CK(cudaMemsetAsync(d_total, 0, 24, st));
  if (d.bound)
    { k_key_max<<<std::min(grid_for((nb + 3) / 4), 4 * sm_count()), 256, 0, st>>>((const uint32_t *)bkeys, nb, d.ctl); vs::note_launch(); }
  { k_join_clear<<<std::min(grid_for(std::max<uint64_t>(tp.cap + 1, d.bound / 4)), cap_grid), 256, 0, st>>>(d, !early); vs::note_launch(); }
  const uint64_t first = std::min<uint64_t>(nb, d.bound ? 512ull * sm_count() : nb);  // rows
  if (first) { k_join_build<<<grid_for(first), 256, 0, st>>>(d, bkeys, ktype, slot_of, 0, first); vs::note_launch(); }
  if (nb > first) { k_join_build<<<grid_for(nb - first), 256, 0, st>>>(d, bkeys, ktype, slot_of, first, nb); vs::note_launch(); }
  struct {
    unsigned long long total;
    uint32_t top, repeated;
  } h{};
  auto probe = [&](int unique_only) {
    if (np) {
      k_join_probe<<<grid_for(np), 256, 0, st>>>(d, pkeys, ktype, np, sums, pcnt, pslot, d_total, unique_only);
      vs::note_launch();
    }
  };
  auto ask = [&]() {  // the rows' number, and the mode
    VS_CK(cudaGetLastError());
    VS_CK(cudaMemcpyAsync(&h, d_total, 16, cudaMemcpyDeviceToHost, st));
    VS_CK(cudaStreamSynchronize(st));
    return VS_OK;
  };
  auto unique = [&]() { return d.bound && h.top < d.bound && !h.repeated; };
  if (early) {
    probe(1);
    VS_TRY(ask());
  }
  if (!early || !unique()) {
    if (early && h.top < d.bound) VS_CK(cudaMemsetAsync(d.t.cnt, 0, 8 * nb, st));  // its slots, not cleared yet
    if (d.bound) { k_join_count<<<std::min(grid_for(nb), cap_grid), 256, 0, st>>>(d, (const uint32_t *)bkeys, slot_of); vs::note_launch(); }
    { k_join_scan<<<std::min(grid_for(tp.cap + 1, 1024), cap_grid), 256, 0, st>>>(d, d.t.cnt, d.t.off, d.tile_off, tp.cap + 1,
                                                                                  nb, d.ctl + 2); vs::note_launch(); }
    if (nb) { k_join_scatter<<<std::min(grid_for(nb), cap_grid), 256, 0, st>>>(d, slot_of, rows_by_key); vs::note_launch(); }
    probe(0);
    { k_join_scan<<<std::min(grid_for(np + 1, 1024), cap_grid), 256, 0, st>>>(d, pcnt, poff, ptile, np, np, d.ctl + 3); vs::note_launch(); }
    VS_TRY(ask());
  }
  *count = h.total;
  const uint64_t rows = std::min<uint64_t>(h.total, max_rows);
  int32_t types[16];
  EmitArgs ea{};
  VS_TRY(join_columns(a, b, build_a, types, &ea));
  vs_flat *f = nullptr;
  VS_TRY(flat_alloc(ea.ncols, types, rows, st, &f));
  for (int i = 0; i < ea.ncols; i++) ea.col[i].dst = f->cols[i];
  ea.poff = poff;
  ea.ptile = ptile;
  ea.pslot = pslot;
  ea.rows_by_key = rows_by_key;
  ea.b = d;
  ea.n_probe = np;
  ea.out_rows = rows;
  int rc = VS_OK;
  if (rows && unique()) {
    rc = exclusive_scan_u64(sums, offs, tiles, st);
    if (rc == VS_OK)
      { k_fk_emit<<<(int)std::min<uint64_t>(tiles, cap_grid), 256, 0, st>>>(ea, (const uint32_t *)pkeys, offs); vs::note_launch(); }
  } else if (rows) {
    k_emit<<<(unsigned)((rows + EMIT_ROWS - 1) / EMIT_ROWS), 256, 0, st>>>(ea);
    vs::note_launch();
  }
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (rc != VS_OK || e != cudaSuccess) {
    vs_flat_free(f);
    return rc != VS_OK ? rc : cuda_fail(e, "hash join", __FILE__, __LINE__);
  }
  *out = f;
  return h.total > max_rows ? fail(VS_ERR_CAPACITY, "join produced %llu rows, bound %llu", h.total,
                                   (unsigned long long)max_rows)
                            : VS_OK;
}

// Count-only Flat x Mat: the flat side's multiplicities against column popcounts.
int count_flat_mat(FlatSide f, const vs_bitmat *m, uint64_t *count, cudaStream_t st) {
  if (f.f->types[f.key] != VS_T_VID) return fail(VS_ERR_ARG, "matrix keys are VIDs; flat key is not");
  Scratch sc{st};
  TablePart tp;
  tp.add(sc, f.f->nrows, false, 1);
  VS_TRY(sc.alloc());
  VS_TRY(tp.clear(sc));
  const Table t = tp.table(sc);
  if (f.f->nrows)
    { k_build<<<grid_for(f.f->nrows), 256, 0, st>>>(t, f.f->cols[f.key], VS_T_VID, f.f->nrows); vs::note_launch(); }
  unsigned long long *d_total = sc.at<unsigned long long>(tp.zeroed);
  if (m->cols)
    { k_count_mat<<<grid_for((uint64_t)m->cols * 32), 256, 0, st>>>(t, m->words, m->cols, m->wpc,
                                                                 m->col_map, d_total); vs::note_launch(); }
  VS_CK(cudaGetLastError());
  return read_total(d_total, count, st);
}

int count_mat_mat(const vs_bitmat *a, const vs_bitmat *b, uint64_t *count, cudaStream_t st) {
  Scratch sc{st};
  const bool direct = !a->col_map && !b->col_map;
  if (direct) {
    sc.add<uint64_t>(1);
    VS_TRY(sc.alloc());
    unsigned long long *d_total = sc.at<unsigned long long>(0);
    VS_CK(cudaMemsetAsync(d_total, 0, 8, st));
    const uint32_t cols = std::min(a->cols, b->cols);
    if (cols)
      { k_count_direct<<<grid_for(cols), 256, 0, st>>>(reinterpret_cast<const uint4 *>(a->words), a->wpc / 2,
                                                      reinterpret_cast<const uint4 *>(b->words), b->wpc / 2, cols,
                                                      a->colnz, b->colnz, d_total); vs::note_launch(); }
    VS_CK(cudaGetLastError());
    return read_total(d_total, count, st);
  }
  TablePart tp;
  tp.add(sc, a->cols, true, 1);
  VS_TRY(sc.alloc());
  VS_TRY(tp.clear(sc));
  const Table t = tp.table(sc);
  if (a->cols) { k_build_cols<<<grid_for(a->cols), 256, 0, st>>>(t, a->col_map, a->cols); vs::note_launch(); }
  unsigned long long *d_total = sc.at<unsigned long long>(tp.zeroed);
  if (b->cols)
    { k_count_mat_mat<<<grid_for((uint64_t)b->cols * 32), 256, 0, st>>>(
        t, a->words, a->cols, a->wpc, b->words, b->cols, b->wpc, b->col_map, direct ? 1 : 0, d_total); vs::note_launch(); }
  VS_CK(cudaGetLastError());
  return read_total(d_total, count, st);
}

}  // namespace jn
}  // namespace vs

// ---------------------------------------------------------------------------
// Allocation-free count-only join.  Its hash table lives in this file-scope
// device array instead of allocated memory; every GPU that loads the library
// holds the array until the process exits.
namespace vs {
namespace jn {

constexpr uint64_t NOALLOC_SLOTS = 1ull << 19;              // hash slots (power of two)
constexpr uint64_t NOALLOC_MAX_BUILD = NOALLOC_SLOTS / 2;   // load factor <= 1/2
// keys [SLOTS + 1] | counts [SLOTS + 1] | total [1]   (8 MiB + 24 B)
constexpr uint64_t NOALLOC_WORDS = 2 * (NOALLOC_SLOTS + 1) + 1;
static __device__ __align__(256) unsigned long long g_noalloc_scratch[NOALLOC_WORDS];

// Device address of the array, looked up once per device with that device
// current (host code may not use the symbol itself as a device pointer).  A
// cached address is checked against the runtime before use: after
// cudaDeviceReset the device's context, and with it the array, is new, and
// the address is looked up again.
int noalloc_scratch(unsigned long long **out) {
  static std::mutex mu;
  static unsigned long long *addr[128] = {};
  int dev = 0;
  VS_CK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 128) return fail(VS_ERR_UNSUPPORTED, "device index %d out of range", dev);
  std::lock_guard<std::mutex> lock(mu);
  if (addr[dev]) {
    cudaPointerAttributes at{};
    if (cudaPointerGetAttributes(&at, addr[dev]) != cudaSuccess || at.type != cudaMemoryTypeDevice ||
        at.device != dev) {
      cudaGetLastError();  // a stale address is not an error of this call
      addr[dev] = nullptr;
    }
  }
  if (!addr[dev]) {
    void *p = nullptr;
    VS_CK(cudaGetSymbolAddress(&p, g_noalloc_scratch));
    addr[dev] = static_cast<unsigned long long *>(p);
  }
  *out = addr[dev];
  return VS_OK;
}

// The previous call's table is still in the array: reset the slots this
// call uses (keys to empty, counts and the total to zero).
__global__ void k_noalloc_clear(unsigned long long *keys, unsigned long long *cnt,
                                unsigned long long *total, uint64_t cap) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i <= cap;
       i += (uint64_t)gridDim.x * blockDim.x) {
    keys[i] = EMPTY;
    cnt[i] = 0;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) *total = 0;
}

// ---------------------------------------------------------------------------
// Batched join counts over the row blocks of one matrix (batched expand
// results): blockIdx.y is the row block; its warps take chunks of RB_CHUNK
// keys in turn.  A key's column slice of the block (nw words) is read by a
// group of G = min(32, pow2 >= nw) lanes, so narrow blocks put several keys
// in one warp.  The table of blocks travels as a kernel parameter.
constexpr int RB_CHUNK = 256;
struct RowBlocks {
  vs_row_block b[VS_MAX_ROW_BLOCKS];
};

__global__ void __launch_bounds__(256) k_count_row_blocks(const __grid_constant__ RowBlocks tab,
                                                          const uint32_t *__restrict__ keys,
                                                          const uint64_t *__restrict__ w, uint32_t wpc,
                                                          uint32_t cols, const uint32_t *__restrict__ colnz,
                                                          unsigned long long *__restrict__ counts) {
  const vs_row_block rb = tab.b[blockIdx.y];
  if (rb.row_end <= rb.row_begin || rb.key_end <= rb.key_begin) return;
  const uint32_t w0 = rb.row_begin >> 6, nw = ((rb.row_end - 1) >> 6) - w0 + 1;
  const uint64_t m_first = ~0ull << (rb.row_begin & 63);
  const uint64_t m_last = ~0ull >> (63 - ((rb.row_end - 1) & 63));
  uint32_t G = 1;
  while (G < 32 && G < nw) G <<= 1;
  const uint32_t lane = threadIdx.x & 31, grp = lane / G, gl = lane % G, ngrp = 32 / G;
  const uint64_t nkeys = rb.key_end - rb.key_begin;
  const uint64_t nwarps = (uint64_t)gridDim.x * (blockDim.x >> 5);
  const uint32_t *kp = keys + rb.key_begin;
  unsigned long long s = 0;
  for (uint64_t base = ((uint64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * RB_CHUNK;
       base < nkeys; base += nwarps * RB_CHUNK) {
    const uint64_t end = min(base + RB_CHUNK, nkeys);
    for (uint64_t k = base + grp; k < end; k += ngrp) {
      const uint32_t key = __ldg(kp + k);
      if (key >= cols || (colnz && !__ldg(colnz + key))) continue;  // no such vertex / empty column
      const uint64_t *col = w + (size_t)key * wpc + w0;
      for (uint32_t j = gl; j < nw; j += G) {
        uint64_t x = __ldg(col + j);
        if (j == 0) x &= m_first;
        if (j == nw - 1) x &= m_last;
        s += __popcll(x);
      }
    }
  }
  block_add(s, counts + blockIdx.y);
}

}  // namespace jn
}  // namespace vs

using namespace vs;
using namespace vs::jn;

extern "C" {

int vs_hash_join(vs_table_ref a, vs_table_ref b, int only_count, uint64_t max_rows,
                 vs_flat **out, uint64_t *count, vs_stream_t stream) {
  if (!count || (!only_count && !out)) return fail(VS_ERR_ARG, "vs_hash_join: null output");
  if ((!a.flat == !a.mat) || (!b.flat == !b.mat))
    return fail(VS_ERR_ARG, "each join operand is exactly one of a flat table or a matrix");
  cudaStream_t st = S(stream);
  if (out) *out = nullptr;
  *count = 0;
  for (const vs_table_ref *r : {&a, &b}) {
    if (r->flat && r->key_col >= r->flat->ncols) return fail(VS_ERR_ARG, "key column out of range");
    // a matrix joins on its column variable (join.cpp:49-71 assert the key is column 1)
    if (r->mat && r->key_col != 1) return fail(VS_ERR_ARG, "a matrix operand joins on column 1");
  }
  if (only_count) {
    if (a.flat && b.flat) return join_flat_flat({a.flat, a.key_col}, {b.flat, b.key_col}, true, 0, nullptr, count, st);
    if (a.flat && b.mat) return count_flat_mat({a.flat, a.key_col}, b.mat, count, st);
    if (a.mat && b.flat) return count_flat_mat({b.flat, b.key_col}, a.mat, count, st);
    return count_mat_mat(a.mat, b.mat, count, st);
  }
  // materialise: matrix operands become (row value, key) pair tables
  vs_flat *fa = nullptr, *fb = nullptr;
  int rc = VS_OK;
  if (a.mat && (rc = bitmat_to_flat(a.mat, st, &fa)) != VS_OK) return rc;
  if (b.mat && (rc = bitmat_to_flat(b.mat, st, &fb)) != VS_OK) {
    vs_flat_free(fa);
    return rc;
  }
  FlatSide sa{a.flat ? a.flat : fa, a.flat ? a.key_col : 1u};
  FlatSide sb{b.flat ? b.flat : fb, b.flat ? b.key_col : 1u};
  rc = join_flat_flat(sa, sb, false, max_rows, out, count, st);
  cudaStreamSynchronize(st);
  vs_flat_free(fa);
  vs_flat_free(fb);
  return rc;
}


// Count-only join without allocating (see the header): the smaller key column
// is the build side; at most NOALLOC_MAX_BUILD rows.
int vs_hash_join_count_noalloc(const void *keys_a, uint64_t na, const void *keys_b, uint64_t nb,
                               int key_type, uint64_t *count, vs_stream_t stream) {
  if (!count || (na && !keys_a) || (nb && !keys_b))
    return fail(VS_ERR_ARG, "vs_hash_join_count_noalloc: null argument");
  if (key_type != VS_T_VID && key_type != VS_T_I64)
    return fail(VS_ERR_ARG, "vs_hash_join_count_noalloc: unknown key type %d", key_type);
  // the kernels read the keys directly: a host pointer is refused before any launch
  for (const void *p : {na ? keys_a : nullptr, nb ? keys_b : nullptr}) {
    if (!p) continue;
    cudaPointerAttributes at{};
    VS_CK(cudaPointerGetAttributes(&at, p));
    if (at.type != cudaMemoryTypeDevice && at.type != cudaMemoryTypeManaged)
      return fail(VS_ERR_ARG, "vs_hash_join_count_noalloc: keys_a and keys_b must be device memory");
  }
  const bool build_a = na < nb;
  const void *bk = build_a ? keys_a : keys_b, *pk = build_a ? keys_b : keys_a;
  const uint64_t nbld = build_a ? na : nb, nprb = build_a ? nb : na;
  if (nbld > NOALLOC_MAX_BUILD)
    return fail(VS_ERR_CAPACITY,
                "vs_hash_join_count_noalloc: the smaller side has %llu rows; the fixed table holds at most "
                "%llu (use vs_hash_join)",
                (unsigned long long)nbld, (unsigned long long)NOALLOC_MAX_BUILD);
  unsigned long long *base = nullptr;
  VS_TRY(noalloc_scratch(&base));
  cudaStream_t st = S(stream);
  Table t{};
  t.cap = ht_capacity(std::max<uint64_t>(nbld, 1));
  t.keys = base;
  t.cnt = base + (NOALLOC_SLOTS + 1);
  unsigned long long *total = base + 2 * (NOALLOC_SLOTS + 1);
  { k_noalloc_clear<<<grid_for(t.cap + 1), 256, 0, st>>>(t.keys, t.cnt, total, t.cap); vs::note_launch(); }
  if (nbld) { k_build<<<grid_for(nbld), 256, 0, st>>>(t, bk, key_type, nbld); vs::note_launch(); }
  if (nprb) { k_probe<<<grid_for(nprb), 256, 0, st>>>(t, pk, key_type, nprb, total); vs::note_launch(); }
  VS_CK(cudaGetLastError());
  VS_CK(cudaMemcpyAsync(count, total, sizeof(unsigned long long), cudaMemcpyDefault, st));
  VS_CK(cudaStreamSynchronize(st));
  return VS_OK;
}

int vs_hash_join_count_row_blocks(const vs_bitmat *m, const uint32_t *keys, const vs_row_block *blocks,
                                  uint32_t nblocks, uint64_t *counts, vs_stream_t stream) {
  if (!m || !blocks || !counts || nblocks == 0)
    return fail(VS_ERR_ARG, "vs_hash_join_count_row_blocks: null argument or no block");
  if (nblocks > VS_MAX_ROW_BLOCKS)
    return fail(VS_ERR_ARG, "%u row blocks; at most %d per call", nblocks, VS_MAX_ROW_BLOCKS);
  if (m->kind != VS_KIND_VARROW || m->col_map)
    return fail(VS_ERR_ARG, "row-block join counts need a VarRow matrix whose columns are vertex ids");
  RowBlocks tab{};
  uint64_t max_keys = 0;
  for (uint32_t q = 0; q < nblocks; q++) {
    const vs_row_block &b = blocks[q];
    if (b.row_begin > b.row_end || b.row_end > m->rows || b.key_begin > b.key_end)
      return fail(VS_ERR_ARG, "row block %u: rows [%u, %u) of %u, keys [%llu, %llu)", q, b.row_begin,
                  b.row_end, m->rows, (unsigned long long)b.key_begin, (unsigned long long)b.key_end);
    tab.b[q] = b;
    max_keys = std::max<uint64_t>(max_keys, b.key_end - b.key_begin);
  }
  if (max_keys && !keys) return fail(VS_ERR_ARG, "vs_hash_join_count_row_blocks: null keys");
  for (const void *p : {(const void *)keys, (const void *)counts}) {
    if (!p) continue;
    cudaPointerAttributes at{};
    VS_CK(cudaPointerGetAttributes(&at, p));
    if (at.type != cudaMemoryTypeDevice && at.type != cudaMemoryTypeManaged)
      return fail(VS_ERR_ARG, "vs_hash_join_count_row_blocks: keys and counts must be device memory");
  }
  cudaStream_t st = S(stream);
  VS_CK(cudaMemsetAsync(counts, 0, sizeof(uint64_t) * nblocks, st));
  if (max_keys == 0 || m->rows == 0) return VS_OK;
  const uint64_t warps_needed = (max_keys + RB_CHUNK - 1) / RB_CHUNK;
  const uint32_t gx = (uint32_t)std::min<uint64_t>((warps_needed + 7) / 8, (uint64_t)sm_count() * 8);
  { k_count_row_blocks<<<dim3(gx, nblocks), 256, 0, st>>>(tab, keys, m->words, m->wpc, m->cols, m->colnz,
                                                          reinterpret_cast<unsigned long long *>(counts));
    vs::note_launch(); }
  VS_CK(cudaGetLastError());
  return VS_OK;
}

}  // extern "C"
