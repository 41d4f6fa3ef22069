// Multi-source bit-matrix expand: VExpand + Expand<DenseVarStackMatrix>
// (src/objects/operator/vexpand.cpp, src/objects/operator/expand.cpp,
// src/include/operator/expand_impl.hh) re-designed for sm_103a.
//
// Data layout in HBM.  Every matrix is vertex-major: vertex v owns W
// consecutive uint64 words (W = ceil(S/64) rounded up to even), bit i of the
// row is source i.  This is the reference's DenseVarStackMatrix with a single
// stack as tall as S (rows padded to 128 instead of 1024), so one hop gathers
// 8W bytes per active edge instead of a padded 128-byte stack slice per stack.
//
// Buffers: two frontier buffers (layer h-1 and layer h ping-pong), the
// visited matrix (Shortest/FindShortest) and the accumulator (the union of
// layers k_min..k_max when it differs from visited).  Each frontier buffer
// has one uint32 flag per vertex with the invariant "flag == 0 => row is
// zero", which lets a hop skip inactive rows and clear only what it wrote
// (flag 2: a non-zero short row kept only in its short-row slot, the buffer
// row being zero; see the short-row notes at the PULL kernels).
//
// Per hop one of three strategies runs; the choice is made ON THE DEVICE by a
// one-block decide kernel from the previous hop's counters, so a whole query
// is a fixed launch sequence that can be captured in a CUDA graph:
//   SPARSE  (vertex, source) pair lists, one atomicOr per (pair, edge): the
//           reference's CSR strategy (expand.cpp:43-131) as an exact
//           bit-matrix update; used from the sources and while frontiers are tiny.
//   PULL    every vertex ORs the rows of its active in-neighbours with 16-byte
//           coalesced loads (sub-warp groups for narrow rows), fused with the
//           visited AND-NOT, the [k_min,k_max] accumulation and the popcounts
//           (dedup_and_update_visit_and_count, bitmap.cpp:1054-1096, and
//           merge_to_MT's union, vexpand.cpp:298-354, folded into the hop).
//           Vertices above the hub threshold are cut into pieces.
//   PUSH    active rows OR-ed into their out-neighbours with 64-bit atomics,
//           followed by a fused dedup/accumulate pass over the touched rows.
#include <algorithm>
#include <atomic>
#include <mutex>
#include <cstring>
#include <vector>

#include "expand_internal.cuh"
#include "picker.cuh"
#include "vs_internal.cuh"

namespace vs {
namespace ex {

constexpr unsigned FULL = 0xffffffffu;

__device__ __forceinline__ unsigned lanemask_lt() {
  unsigned m;
  asm volatile("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

template <typename T> __device__ __forceinline__ T warp_sum(T v) {
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
  return v;
}

// Block-wide sum of per-thread counters, one atomic per block.
__device__ __forceinline__ void block_add(unsigned long long v, unsigned long long *dst) {
  __shared__ unsigned long long part[32];
  v = warp_sum(v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
    v = threadIdx.x < (blockDim.x >> 5) ? part[threadIdx.x] : 0ull;
    v = warp_sum(v);
    if (threadIdx.x == 0 && v) atomicAdd(dst, v);
  }
}

// ---------------------------------------------------------------------------
// Zero the flagged rows of a buffer and their flags.
__device__ __forceinline__ void clear_flagged(uint4 *__restrict__ buf, uint32_t *__restrict__ flag, uint32_t V,
                                              uint32_t Q) {
  const int lane = threadIdx.x & 31;
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  // four flags per lane (16-byte loads of the 16-byte aligned flag array):
  // a warp step covers 128 vertices, so the scan is a quarter as many
  // dependent loads; flag 2 means the row lives in its slot (buffer row zero)
  uint4 *flag4 = reinterpret_cast<uint4 *>(flag);
  const uint32_t nq = V / 4;
  for (uint32_t base = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * 32; base < nq; base += warps * 32) {
    const uint32_t g = base + lane;
    const uint4 f = g < nq ? flag4[g] : make_uint4(0, 0, 0, 0);
    if (f.x | f.y | f.z | f.w) flag4[g] = make_uint4(0, 0, 0, 0);
    const uint32_t fv[4] = {f.x, f.y, f.z, f.w};
    if (Q <= 8) {
      // narrow rows: the 128 rows are one range, its flagged cells stored by all
      // lanes (a row at a time left most lanes idle: 1M rows of 16 bytes 43 -> 6 us)
      unsigned m[4];
#pragma unroll
      for (int k = 0; k < 4; k++) m[k] = __ballot_sync(FULL, fv[k] == 1);
      if (!(m[0] | m[1] | m[2] | m[3])) continue;
      uint4 *rows = buf + (size_t)base * 4 * Q;
      uint32_t r = lane / Q, q = lane % Q;  // cell lane + 32 i: row r, uint4 q
      const uint32_t dr = 32 / Q, dq = 32 % Q;
      for (uint32_t i = lane; i < 128 * Q; i += 32) {
        const unsigned mk = (r & 2) ? (r & 1 ? m[3] : m[2]) : (r & 1 ? m[1] : m[0]);
        if (mk >> (r >> 2) & 1u) rows[i] = make_uint4(0, 0, 0, 0);
        r += dr;
        q += dq;
        if (q >= Q) {
          q -= Q;
          r++;
        }
      }
      continue;
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
      unsigned m = __ballot_sync(FULL, fv[k] == 1);
      while (m) {
        const int b = __ffs(m) - 1;
        m &= m - 1;
        uint4 *row = buf + (size_t)((base + b) * 4u + k) * Q;
        for (uint32_t q = lane; q < Q; q += 32) row[q] = make_uint4(0, 0, 0, 0);
      }
    }
  }
  if (blockIdx.x == 0 && threadIdx.x < 32) {  // the last V % 4 vertices
    for (uint32_t v = nq * 4; v < V; v++) {
      const uint32_t f = flag[v];
      if (f == 1)
        for (uint32_t q = lane; q < Q; q += 32) buf[(size_t)v * Q + q] = make_uint4(0, 0, 0, 0);
      __syncwarp();
      if (lane == 0 && f) flag[v] = 0;
    }
  }
}

// Run start: the rows the previous run left in both frontier buffers and in the
// result (NULL: none), and the counter block (n 16-byte words).
__global__ void __launch_bounds__(256) k_run_start(uint4 *buf0, uint32_t *flag0, uint4 *buf1, uint32_t *flag1, uint4 *res,
                                                   uint32_t *resflag, uint32_t V, uint32_t Q, uint4 *ctr, uint32_t n) {
  vs::grid_wait();
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    ctr[i] = make_uint4(0, 0, 0, 0);
  clear_flagged(buf0, flag0, V, Q);
  clear_flagged(buf1, flag1, V, Q);
  if (res) clear_flagged(res, resflag, V, Q);
}

// Layer 0 (ExpandStatus::init_first_m_layer, expand_impl.hh:252-277).
__device__ __forceinline__ int degree_bin(unsigned long long d) {
  return min(pk::NHIST - 1, 63 - __clzll((long long)(d + 1)));
}

__global__ void k_seed(SeedArgs a) {
  vs::grid_wait();
  __shared__ unsigned s_hist[pk::NHIST];  // hop 1's frontier statistics (a.stats)
  if (threadIdx.x < pk::NHIST) s_hist[threadIdx.x] = 0;
  __syncthreads();
  unsigned long long pe = 0, nv = 0, ae = 0;
  if (blockIdx.x == 0 && threadIdx.x == 0) {  // counters set on the device: the run has no host copies
    a.ctr->multislice = a.multislice;
    a.ctr->hop[0].pairs = a.S;
    a.ctr->hop[0].new_bits = a.S;
    if (a.rowk && a.rowk[1]) atomicOr(&a.ctr->error, 2);  // a device-set row limit exceeded k_max
  }
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < a.S; i += gridDim.x * blockDim.x) {
    uint32_t v = a.sources[i];
    if (v >= a.V) {  // reported as VS_ERR_ARG; the pair stays in range
      a.ctr->error = 1;
      a.pairs0[i] = make_uint2(0, i);
      a.pdeg0[i] = 0;
      continue;
    }
    size_t idx = (size_t)v * a.W + (i >> 6);
    unsigned long long bit = 1ull << (i & 63);
    atomicOr((unsigned long long *)&a.buf0[idx], bit);
    const bool first = atomicOr(&a.flag0[v], 1u) == 0;
    if (first) nv++;
    if (a.vis) atomicOr((unsigned long long *)&a.vis[idx], bit);
    if (a.acc) atomicOr((unsigned long long *)&a.acc[idx], bit);
    if ((a.vis && a.res_vis) || a.acc) a.resflag[v] = 1;
    a.pairs0[i] = make_uint2(v, i);
    unsigned long long d = 0;
    _Pragma("unroll") for (int l = 0; l < 2; l++) if (l < a.out.n) d += (unsigned long long)(a.out.off[l][v + 1] - a.out.off[l][v]);
    a.pdeg0[i] = d;
    pe += d;
    if (a.stats && first) {  // each distinct source vertex once, as the stats pass counts rows
      ae += d;
      atomicAdd(&s_hist[degree_bin(d)], 1u);
    }
  }
  block_add(pe, &a.ctr->hop[0].pair_edges);
  block_add(nv, &a.ctr->hop[0].active_vertices);
  if (a.stats) {
    block_add(ae, &a.ctr->hop[1].active_edges);
    if (threadIdx.x < pk::NHIST && s_hist[threadIdx.x])
      atomicAdd(&a.ctr->hop[1].hist[threadIdx.x], (unsigned long long)s_hist[threadIdx.x]);
  }
}

// FindShortest bookkeeping before hop 1 (VExpand::before_execution, vexpand.cpp:179-195).
__global__ void k_dist_init(const uint32_t *__restrict__ src, const uint32_t *__restrict__ tgt,
                            int32_t *__restrict__ dist, uint32_t S, uint32_t V, Ctr *ctr) {
  vs::grid_wait();
  unsigned long long f = 0;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < S; i += gridDim.x * blockDim.x) {
    if (tgt[i] >= V) ctr->error = 1;
    bool eq = src[i] == tgt[i];
    dist[i] = eq ? 0 : -1;
    f += eq;
  }
  block_add(f, &ctr->found);
}

// with_distance export: layer h (the frontier buffer just written) into its
// own zeroed matrix, flagged rows only; a hop that did not run copies nothing.
__global__ void k_copy_layer(const uint4 *__restrict__ buf, const uint32_t *__restrict__ flag, uint4 *__restrict__ out,
                             uint32_t V, uint32_t Q, const Ctr *ctr, int h) {
  vs::grid_wait();
  if (h > 0 && ctr->hop[h].strategy == 0) return;
  const int lane = threadIdx.x & 31;
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  for (uint32_t base = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * 32; base < V; base += warps * 32) {
    const uint32_t v = base + lane;
    unsigned m = __ballot_sync(FULL, v < V && flag[v]);
    while (m) {
      const int b = __ffs(m) - 1;
      m &= m - 1;
      const size_t row = (size_t)(base + b) * Q;
      for (uint32_t q = lane; q < Q; q += 32) out[row + q] = buf[row + q];
    }
  }
}

// Per-hop row masks of batched queries from per-row hop limits: word w of
// hop h has bit r set when row 64w+r may still grow at hop h.
__global__ void __launch_bounds__(256) k_row_mask(const uint8_t *__restrict__ lim, uint32_t n, uint32_t K, uint32_t W,
                                                  uint64_t *__restrict__ hmask, uint32_t *rowk) {
  const uint32_t lane = threadIdx.x & 31, w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (w >= W) return;  // a warp per word: a lane's two rows, a ballot per hop
  const uint32_t i = w * 64 + lane, j = i + 32;
  const uint32_t a = i < n ? lim[i] : 0u, b = j < n ? lim[j] : 0u, top = __reduce_max_sync(FULL, max(a, b));
  for (uint32_t h = 0; h <= K; h++) {
    const unsigned lo = __ballot_sync(FULL, h && a >= h), hi = __ballot_sync(FULL, h && b >= h);
    if (lane == 0) hmask[(size_t)h * W + w] = (uint64_t)lo | (uint64_t)hi << 32;
  }
  if (lane == 0) {
    if (top) atomicMax(&rowk[0], min(top, K));
    if (top > K) rowk[1] = 1;
  }
}

// Row flags as bits in a block's shared memory: up to BITS_MAX_V vertices (160 KB; the
// rest of the SM's 228 KB stays L1).
constexpr uint32_t BITS_MAX_V = 160 * 1024 * 8;
constexpr uint32_t BITS_MIN_V = 128 * 1024;
constexpr uint64_t BITS_MIN_EDGES = 16ull << 20;
inline size_t bits_smem(uint32_t V) { return (size_t)((V + 127) / 128) * 16; }

// One block of 256 threads: early-stop checks of hop h-1 (VExpand::after_child,
// vexpand.cpp:222-284), the fixed planner's choice for hop h, and — when a
// picker is loaded or features are logged — the feature vector of hop h and
// the picker network's choice.
__global__ void __launch_bounds__(256) k_decide(DecideArgs a) {
  __shared__ float f[pk::NF], out[pk::NO];
  __shared__ int s_run, s_choice, s_pairs_ok;
  const int t = threadIdx.x;
  Ctr *c = a.ctr;
  HopCtr &prev = c->hop[a.h - 1];
  HopCtr &cur = c->hop[a.h];
  const bool use_picker = a.picker && a.picker_on && a.forced == 0;
  // the network's parameters load while thread 0 reads the counters
  const __nv_bfloat16 *w = use_picker ? pk::mlp_stage(a.picker) : nullptr;
  vs::grid_wait();
  if (t == 0) {
    if (!c->done && a.rowk && (uint32_t)a.h > a.rowk[0]) c->done = 1;  // every row is past its last hop
    if (!c->done && a.h >= 2) {
      if (a.path != VS_PATH_ANY && prev.new_bits == 0) c->done = 1;
      if (a.path == VS_PATH_FIND_SHORTEST && c->found >= a.S) c->done = 1;
    }
    s_run = !c->done;
    s_choice = 0;
    s_pairs_ok = 0;
    if (s_run) {
      c->hops_run = a.h;
      const bool pairs_ok = (a.h == 1) || (prev.strategy == ST_SPARSE && !prev.overflow &&
                                           prev.pairs <= a.pair_cap);
      s_pairs_ok = pairs_ok;
      int s = a.forced;
      if (s == ST_SPARSE && !pairs_ok) s = ST_PULL;
      if (s == 0) {
        // fixed planner: pair lists while their edge work is a small fraction
        // of a dense pass, then push while few rows are active, then pull
        const double pe = (double)prev.pair_edges;
        if (pairs_ok && pe < (double)a.E * a.sparse_frac)
          s = ST_SPARSE;
        else if ((double)prev.active_vertices < (double)a.V * a.push_frac && prev.strategy != 0)
          s = ST_PUSH;
        else
          s = ST_PULL;
      }
      s_choice = s;
    }
  }
  __syncthreads();
  if (!s_run) {
    if (t == 0) cur.strategy = 0;
    return;
  }
  if (use_picker || a.log_features) {
    if (t == 0) {
      pk::HopFeatIn in;
      in.S = (float)a.S;
      in.V = (float)a.V;
      in.E = (float)a.E;
      in.W = (float)a.W;
      in.h = (float)a.h;
      in.k_min = (float)a.k_min;
      in.k_max = (float)a.k_max;
      in.new_bits_prev = (float)prev.new_bits;
      in.active_prev = (float)prev.active_vertices;
      unsigned long long vis = 0;
      for (int i = 0; i < a.h; i++) vis += c->hop[i].new_bits;
      in.visited_bits = (float)vis;
      in.active_edges = (float)cur.active_edges;
      in.pair_edges = s_pairs_ok ? (float)prev.pair_edges : 0.f;
      in.pairs_ok = (float)s_pairs_ok;
      in.shortest = a.path != VS_PATH_ANY ? 1.f : 0.f;
      in.both = (float)a.both;
      in.hist = cur.hist;
      pk::hop_features(in, f);
      if (a.log_features)
        for (int i = 0; i < pk::NF; i++) c->feat[a.h][i] = f[i];
    }
    __syncthreads();
    // one choice left (no pair list, no PUSH in the plan): PULL without the network
    if (use_picker && (s_pairs_ok || a.push_ok)) {
      pk::mlp_run(w, f, out);
      if (t == 0) {
        int best = -1;
        for (int k = 0; k < pk::NO; k++) {
          const int st = pk::class_to_strategy(k);
          if (st == ST_SPARSE && !s_pairs_ok) continue;  // no pair list to expand from
          if (st == ST_PUSH && !a.push_ok) continue;      // the plan launches no PUSH kernels
          if (best < 0 || out[k] > out[best]) best = k;
        }
        s_choice = pk::class_to_strategy(best);
      }
    }
  }
  if (t == 0) {
    cur.strategy = s_choice;
    // short mode where the hop costs less, in ps fitted on GB300 to 1,920 hops of 2,048
    // to 30,000 sources over power-law, uniform and R-MAT graphs of 100K to 10M vertices,
    // each hop timed dense, from words and from slots (the rule's choices take 1% longer
    // than the best of the three; with prices taken at 1M vertices and more they took up
    // to 2.1 times as long at 200K to 1M).  A dense hop pays 11 to 24 per list entry for
    // neighbour and flag (with the row's lanes) and 0.88 per word of every active row;
    // short mode 12.5 per entry, 19 per id read from words (3 on a last hop, which keeps no
    // lists; 33 where every target is searched for its bits), 1.1 per id read from slots
    // of 32 bytes (wider ones 0.75, and 14 per entry) and 3.1 per word of the target rows
    // then searched (none on a last hop), and 0.9 per word of a row too long for a slot.
    bool sp = false, slots = false, lng = false;
    if (s_choice == ST_PULL && a.short_min > 0 && !c->multislice) {
      const bool counted = prev.strategy == ST_PULL;  // ... its layer's words, slots and degrees
      const float act = (float)prev.active_vertices, V = (float)a.V, E = (float)a.E * (a.both ? 2 : 1), W = (float)a.W;
      const float ids = prev.strategy == ST_PUSH ? E * ((float)prev.new_bits / V) : (float)prev.pair_edges;
      float rows, longs = 0, so = 0;  // edges leaving non-empty rows, rows too long for a slot, and rows within one
      if (counted) {
        rows = (float)prev.row_out;
        so = (float)prev.short_out;
        longs = (float)(prev.row_out - prev.short_out);
      } else {
        rows = ids * (act / fmaxf(1.f, (float)prev.new_bits));
      }
      const float t_long = 0.9f * W * longs, held = a.W <= 64 ? 15.f : a.W <= 128 ? 31.f : 63.f;  // ids a slot holds
      const float t_words = 12.5f * E + (a.last ? 3.f : a.gen ? 33.f : 19.f) * ids + t_long;
      const float t_slots = (a.W <= 64 ? 12.5f : 14.f) * E + (a.W <= 64 ? 1.1f : 0.75f) * fminf(ids, held * so) +
                            (a.last ? 0.f : 3.1f * V * W) + t_long;
      slots = counted && t_slots < t_words;
      if (a.short_min > 1.0) {
        sp = true;
      } else if (!counted || (double)(prev.short_rows & 0xFFFFFFFFull) >= a.short_min * (double)prev.active_vertices) {
        const float flag = act >= 0.9f * V ? 11.f : a.W <= 32 ? 16.f : 24.f;
        sp = (slots ? t_slots : t_words) < 0.8f * (flag * E + 0.88f * W * rows);
      }
      // more than half a slot of ids per target: its new row will often be long
      lng = ids > 1.2f * V * (held + 1.f);
    }
    cur.short_pull = sp;
    // row flags as bits where they save loads: below 9 in 10 active vertices for rows of
    // more than a sector.  A narrower row is loaded as fast as its flag, so only with
    // under half of the list entries active: counted after SPARSE; after PULL a fifth
    // of the vertices (30% of an R-MAT's vertices hold 90% of the entries: 7% slower).
    // Never at hop 1, whose layer is the sources.
    bool bits = s_choice == ST_PULL && !sp && a.bits_ok && a.h > 1;
    if (bits) {
      const float act = (float)prev.active_vertices, V = (float)a.V;
      if (a.W > 2)
        bits = act < 0.9f * V;
      else if (prev.strategy == ST_SPARSE)
        bits = (float)prev.pair_edges * act < 0.5f * (float)a.E * (a.both ? 2 : 1) * (float)prev.new_bits;
      else
        bits = act < 0.2f * V;
    }
    cur.bits = bits;
    cur.short_slots = sp && slots;
    cur.short_long = sp && lng;
  }
}

// Per-hop frontier statistics of layer h-1: E_active (out-degrees of its
// non-zero rows) and the log2(out-degree + 1) histogram of those rows.
// Layers written by the seed or by a SPARSE hop already have these counts
// (counted as their rows became non-zero), so the pass exits at once; so it
// does when only the picker reads them (picker_only) and the hop has a single
// choice: no pair list after a PULL or PUSH hop, and no PUSH in the plan.
__global__ void k_hop_stats(const uint32_t *__restrict__ flagF, Lists out, uint32_t V, Ctr *ctr, int h,
                            int picker_only, int push_ok) {
  vs::grid_wait();
  if (ctr->done || h == 1 || ctr->hop[h - 1].strategy == ST_SPARSE) return;
  if (picker_only && !push_ok) return;
  __shared__ unsigned long long hist[pk::NHIST];
  if (threadIdx.x < pk::NHIST) hist[threadIdx.x] = 0;
  __syncthreads();
  unsigned long long s = 0;
  // warp-uniform loop; lanes with the same bin add once through their leader
  for (uint32_t v0 = (blockIdx.x * blockDim.x + threadIdx.x) & ~31u; v0 < V; v0 += gridDim.x * blockDim.x) {
    const uint32_t v = v0 + (threadIdx.x & 31);
    int b = -1;
    if (v < V && flagF[v]) {
      unsigned long long d = 0;
      _Pragma("unroll") for (int l = 0; l < 2; l++) if (l < out.n) d += (unsigned long long)(out.off[l][v + 1] - out.off[l][v]);
      s += d;
      b = degree_bin(d);
    }
    const unsigned peers = __match_any_sync(FULL, b);
    if (b >= 0 && (peers & lanemask_lt()) == 0) atomicAdd(&hist[b], (unsigned long long)__popc(peers));
  }
  __syncthreads();
  if (threadIdx.x < pk::NHIST && hist[threadIdx.x]) atomicAdd(&ctr->hop[h].hist[threadIdx.x], hist[threadIdx.x]);
  block_add(s, &ctr->hop[h].active_edges);
}

// SPARSE: (vertex u, source i) pairs of layer h-1; every out-neighbour v gets
// bit i.  Shortest dedups through the visited bit (atomicOr returns the old
// word), Any through the next-layer bit.  New pairs form layer h's list.
// The work is balanced over edges, not pairs: a prefix sum of the pairs'
// out-degrees (k_pscan) lays all their out-lists end to end, and each warp
// takes fixed chunks of that edge range, so a pair on a 50k-degree hub is
// spread over many warps instead of serialising one.
constexpr int SPARSE_CHUNK = 256;  // edges per warp task at most
constexpr int SPARSE_K = 2;        // edges per lane per round

// Pairs the SPARSE hop h scans (0 when the hop runs another strategy).
__device__ __forceinline__ uint64_t scan_len(const Ctr *ctr, int h, uint64_t cap) {
  if (ctr->hop[h].strategy != ST_SPARSE) return 0;
  const unsigned long long npr = ctr->hop[h - 1].pairs;
  return npr < cap ? npr : cap;
}

// Exclusive prefix of the pairs' out-degrees in two levels, in one launch: doff
// within tiles of 1,024 pairs, and by the block that finishes last the tiles' starts
// (bsum, the total after them).  A reader adds the two, which costs a load beside
// the one it waits for anyway and saves a pass and two launches.
__device__ __forceinline__ unsigned long long block_scan4(unsigned long long (&v)[4], unsigned long long *wt) {
  // v becomes the exclusive prefix over the block's 1,024 values; returns their sum
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  unsigned long long run = v[0] + v[1] + v[2] + v[3], incl = run;
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
}

__global__ void __launch_bounds__(256) k_pscan(const unsigned long long *__restrict__ pdeg,
                                               unsigned long long *__restrict__ doff,
                                               unsigned long long *__restrict__ bsum, Ctr *ctr, int h, uint64_t cap) {
  vs::grid_wait();
  const uint64_t np = scan_len(ctr, h, cap);
  const uint64_t nb = (np + 1023) / 1024;
  if (blockIdx.x >= nb) return;
  __shared__ unsigned long long wt[8];
  __shared__ bool s_last;
  const int t = threadIdx.x;
  unsigned long long v[4];
  for (uint64_t b = blockIdx.x; b < nb; b += gridDim.x) {
    const uint64_t base = b * 1024 + (uint64_t)t * 4;
#pragma unroll
    for (int k = 0; k < 4; k++) v[k] = base + k < np ? pdeg[base + k] : 0ull;
    const unsigned long long sum = block_scan4(v, wt);
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (base + k < np) doff[base + k] = v[k];
    if (t == 0) bsum[b] = sum;
  }
  __threadfence();
  __syncthreads();
  const uint64_t blocks = nb < gridDim.x ? nb : gridDim.x;
  if (t == 0) s_last = atomicAdd(&ctr->hop[h].scan_done, 1u) == blocks - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  unsigned long long carry = 0;
  for (uint64_t b0 = 0; b0 < nb; b0 += 1024) {
    const uint64_t base = b0 + (uint64_t)t * 4;
#pragma unroll
    for (int k = 0; k < 4; k++) v[k] = base + k < nb ? __ldcg(bsum + base + k) : 0ull;
    const unsigned long long sum = block_scan4(v, wt);
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (base + k < nb) bsum[base + k] = carry + v[k];
    carry += sum;
  }
  if (t == 0) bsum[nb] = carry;
}

// First edge of pair p in the layer's edge range.
__device__ __forceinline__ unsigned long long pair_start(const unsigned long long *__restrict__ doff,
                                                         const unsigned long long *__restrict__ bsum, uint64_t p) {
  return doff[p] + bsum[p >> 10];
}

__device__ __forceinline__ unsigned long long out_degree(const Lists &L, uint32_t v) {
  unsigned long long d = 0;
  _Pragma("unroll") for (int l = 0; l < 2; l++) if (l < L.n) d += (unsigned long long)(L.off[l][v + 1] - L.off[l][v]);
  return d;
}

// Largest p in [0, np) with pair_start(p) <= x for x0 (lanes 0-15) and x1 (lanes
// 16-31), starts ascending from 0 <= x: each step a half-warp probes
// 15 positions spread over its range at once and keeps the part between the
// last probe at or below x and the next, so a range shrinks 16-fold per
// dependent load instead of 2-fold.  Every lane receives both answers.
__device__ __forceinline__ void owner_pairs(const unsigned long long *__restrict__ doff,
                                            const unsigned long long *__restrict__ bsum, uint64_t np,
                                            unsigned long long x0, unsigned long long x1, int lane, uint64_t &p0,
                                            uint64_t &p1) {
  const int hl = lane & 15;
  const unsigned long long x = lane < 16 ? x0 : x1;
  uint64_t lo = 0, hi = np;  // doff[lo] <= x, and doff[hi] > x unless hi == np
  while (__any_sync(FULL, hi - lo > 1)) {
    const uint64_t span = hi - lo;
    const uint64_t pos = lo + (span * (uint64_t)hl + 15) / 16;  // probe hl; probe 0 is lo itself
    const bool ok = span > 1 && (hl == 0 || (pos < hi && pair_start(doff, bsum, pos) <= x));
    const unsigned b = __ballot_sync(FULL, ok);
    const unsigned half = lane < 16 ? (b & 0xFFFFu) : (b >> 16);
    if (span > 1) {
      const int k = 31 - __clz(half);
      const uint64_t nhi = k == 15 ? hi : lo + (span * (uint64_t)(k + 1) + 15) / 16;
      lo = lo + (span * (uint64_t)k + 15) / 16;
      hi = nhi < hi ? nhi : hi;
    }
  }
  p0 = __shfl_sync(FULL, lo, 0);
  p1 = __shfl_sync(FULL, lo, 16);
}

__global__ void __launch_bounds__(256, 4) k_sparse(SparseArgs a) {
  vs::grid_wait();
  Ctr *c = a.ctr;
  if (c->hop[a.h].strategy != ST_SPARSE) return;
  __shared__ uint2 s_new[8][SPARSE_CHUNK];  // a warp's new pairs of its current chunk
  __shared__ unsigned s_hist[pk::NHIST];    // hop h+1's frontier statistics (a.stats)
  if (threadIdx.x < pk::NHIST) s_hist[threadIdx.x] = 0;
  __syncthreads();
  const unsigned long long np_raw = c->hop[a.h - 1].pairs;
  const uint64_t np = np_raw < a.cap ? np_raw : a.cap;
  const unsigned long long T = np ? a.bsum[(np + 1023) / 1024] : 0ull;
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const uint64_t warps = (uint64_t)gridDim.x * (blockDim.x >> 5);
  // one round of edges per task while that leaves warps idle (a task's rounds are
  // one dependent chain of misses after the other: 10k edges 30 -> 15 us)
  const uint32_t chunk = T < warps * 32 * SPARSE_K * 2 ? 32 * SPARSE_K : SPARSE_CHUNK;
  const uint64_t nchunks = (T + chunk - 1) / chunk;
  unsigned long long nb = 0, nv = 0, pe = 0, ae = 0;
  for (uint64_t ck = (uint64_t)blockIdx.x * (blockDim.x >> 5) + wib; ck < nchunks; ck += warps) {
    const unsigned long long e0 = ck * chunk;
    const unsigned long long e1 = min(e0 + chunk, T);
    // pairs owning the chunk's first and last edge: largest p with doff[p] <= e,
    // both found at once by a 16-way search per half-warp
    uint64_t plo, phi;
    owner_pairs(a.doff, a.bsum, np, e0, e1 - 1, lane, plo, phi);
    uint32_t nloc = 0;  // new pairs of this chunk so far (s_new)
    // the chunk's pairs 32 at a time: lane j holds pair g0 + j (its first
    // edge, source id, and its vertex's list starts and first-list length),
    // and an edge of the group's range finds its pair by a shuffle search over
    // the lanes' first edges instead of loading it
    for (uint64_t g0 = plo; g0 <= phi; g0 += 32) {
      unsigned long long dj = ~0ull;  // lanes past the last pair never own an edge
      uint32_t pi = 0;
      int64_t pb0 = 0, pd0 = 0, pb1 = 0;
      if (g0 + lane <= phi) {
        dj = pair_start(a.doff, a.bsum, g0 + lane);
        const uint2 pr = a.pin[g0 + lane];
        pi = pr.y;
        pb0 = a.out.off[0][pr.x];
        pd0 = a.out.off[0][pr.x + 1] - pb0;
        if (a.out.n > 1) pb1 = a.out.off[1][pr.x];
      }
      // the group's edges inside the chunk
      const unsigned long long d0j = __shfl_sync(FULL, dj, 0);
      const unsigned long long gs = d0j > e0 ? d0j : e0;
      unsigned long long ge = e1;
      if (g0 + 32 <= phi) {
        const unsigned long long nx = pair_start(a.doff, a.bsum, g0 + 32);
        ge = nx < e1 ? nx : e1;
      }
      // SPARSE_K edges per lane per round, each phase issued for all of them
      // before the next: the adjacency loads, then the returning atomics on
      // the visited (or next-layer) words, then the row flags, so a lane keeps
      // SPARSE_K dependent chains in flight instead of one
      for (unsigned long long eb = gs; eb < ge; eb += 32 * SPARSE_K) {
        uint32_t v[SPARSE_K], i[SPARSE_K];
        bool act[SPARSE_K];
#pragma unroll
        for (int k = 0; k < SPARSE_K; k++) {
          const unsigned long long e = eb + k * 32 + lane;
          int own = 0;  // the last pair whose first edge is at or below e (starts ascend with the lane)
#pragma unroll
          for (int step = 16; step; step >>= 1)
            if (__shfl_sync(FULL, dj, own + step) <= e) own += step;
          i[k] = __shfl_sync(FULL, pi, own);
          const int64_t b0 = __shfl_sync(FULL, pb0, own);
          const int64_t d0 = __shfl_sync(FULL, pd0, own);
          const int64_t b1 = __shfl_sync(FULL, pb1, own);
          const unsigned long long j = e - __shfl_sync(FULL, dj, own);  // the edge's index in its pair's out-lists
          v[k] = 0;
          act[k] = e < ge && (!a.hmask || ((__ldg(a.hmask + (i[k] >> 6)) >> (i[k] & 63)) & 1ull));
          if (act[k]) v[k] = (int64_t)j < d0 ? a.out.adj[0][b0 + j] : a.out.adj[1][b1 + (int64_t)j - d0];
        }
        unsigned long long old[SPARSE_K];
#pragma unroll
        for (int k = 0; k < SPARSE_K; k++) {
          old[k] = ~0ull;  // an inactive edge sets nothing
          if (act[k]) {
            const size_t idx = (size_t)v[k] * a.W + (i[k] >> 6);
            // Shortest dedups through the visited bit, Any through the next-layer bit
            old[k] = atomicOr(a.shortest ? &a.vis[idx] : &a.N[idx], 1ull << (i[k] & 63));
          }
        }
        bool fresh[SPARSE_K];
#pragma unroll
        for (int k = 0; k < SPARSE_K; k++) {
          fresh[k] = !((old[k] >> (i[k] & 63)) & 1ull);
          if (fresh[k]) {
            const size_t idx = (size_t)v[k] * a.W + (i[k] >> 6);
            const unsigned long long bit = 1ull << (i[k] & 63);
            if (a.shortest && !a.last && !a.defer) atomicOr(&a.N[idx], bit);
            if (a.acc_on) atomicOr(&a.acc[idx], bit);
            nb++;
          }
        }
        bool first[SPARSE_K];
#pragma unroll
        for (int k = 0; k < SPARSE_K; k++) {
          // a last layer's rows stay zero in the buffer (flag 2: the run start skips them)
          first[k] = fresh[k] && atomicOr(&a.flagN[v[k]], a.last ? 2u : 1u) == 0;
          nv += first[k];
          // the result column is marked once per row and hop, by the bit that made the row non-zero
          if (first[k] && (a.res_vis || a.acc_on)) a.resflag[v[k]] = 1;
        }
        // the chunk's new pairs gather in shared memory (one list append per chunk);
        // bit 31 of the source id (S < 2^31) marks the pair that made its row non-zero
#pragma unroll
        for (int k = 0; k < SPARSE_K; k++) {
          const unsigned m = __ballot_sync(FULL, fresh[k]);
          if (fresh[k])
            s_new[wib][nloc + __popc(m & lanemask_lt())] = make_uint2(v[k], i[k] | (first[k] ? 0x80000000u : 0u));
          nloc += __popc(m);
        }
      }
    }
    __syncwarp();
    if (nloc && a.last) {  // a last layer's pairs are counted, not kept
      if (lane == 0) atomicAdd(&c->hop[a.h].pairs, (unsigned long long)nloc);
    } else if (nloc) {  // append the chunk's new pairs (with their out-degrees) to layer h's list
      unsigned long long base = 0;
      if (lane == 0) base = atomicAdd(&c->hop[a.h].pairs, (unsigned long long)nloc);
      base = __shfl_sync(FULL, base, 0);
      for (uint32_t j = lane; j < nloc; j += 32) {
        const uint2 pf = s_new[wib][j];
        const uint2 pr = make_uint2(pf.x, pf.y & 0x7FFFFFFFu);
        const unsigned long long d = out_degree(a.out, pr.x);
        pe += d;
        if (a.stats && (pf.y >> 31)) {  // each row of layer h once, as the stats pass counts them
          ae += d;
          atomicAdd(&s_hist[degree_bin(d)], 1u);
        }
        const unsigned long long slot = base + j;
        if (slot < a.cap) {
          a.pout[slot] = pr;
          a.pdeg_out[slot] = d;
        } else {
          c->hop[a.h].overflow = 1;
          // a deferred row gets the bit a full list cannot hold
          if (a.defer) atomicOr(&a.N[(size_t)pr.x * a.W + (pr.y >> 6)], 1ull << (pr.y & 63));
        }
      }
      __syncwarp();
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) c->hop[a.h].work_edges = T;
  block_add(nb, &c->hop[a.h].new_bits);
  block_add(nv, &c->hop[a.h].active_vertices);
  block_add(pe, &c->hop[a.h].pair_edges);
  if (a.stats) {
    block_add(ae, &c->hop[a.h + 1].active_edges);
    if (threadIdx.x < pk::NHIST && s_hist[threadIdx.x])
      atomicAdd(&c->hop[a.h + 1].hist[threadIdx.x], (unsigned long long)s_hist[threadIdx.x]);
  }
}

// ---------------------------------------------------------------------------
// Short rows.  In the later hops of a many-source expand over a power-law
// graph most frontier rows hold a handful of sources, and a whole-row gather
// then moves mostly zero words.  Every PULL hop with a successor therefore
// also writes, for every vertex, a tiny word (uint32: the ids of a row of one
// or two bits, else its saturated bit count) and a slot of
// slot_n uint16 (entry 0: the count; entries 1..count: the ids, for up to
// slot_n - 1 bits; slot_n = 16, 32 or 64 as the rows are up to 512 B, 1 KB or
// wider).  A later PULL hop in short mode reads, per in-neighbour, either its
// tiny word (word mode: 4 bytes per vertex, an array L2 can hold, loaded with
// an evict-last hint; the slot follows only for rows of more than TINY_MAX
// bits) or its slot alone (slot mode, for frontiers of mostly longer rows):
// count 0 is an empty row, short rows OR their ids into a per-warp
// shared-memory row with 32-bit atomics, and only longer rows are gathered
// whole (see the kernel).  Short rows of a layer with a successor stay in their slots only
// (flag 2, buffer row zero) unless the layer's rows are read directly;
// k_hop_prep writes them out before a hop that reads rows.  Layers
// written by SPARSE or the seed get their words and slots from the hop's
// pair list (k_pairs_slots, k_short_index), layers written by PUSH or an overflowed SPARSE hop
// from their rows (k_short_index), when the next hop reads them.
// A tiny word is 0 for an empty row; otherwise its top two bits are a class:
// 1 = one id in bits 0..14, 2 = two ids in bits 0..14 and 15..29, 3 = the
// row's bit count (saturated at 0xFFFF) in bits 0..15, its ids in the slot
// when the count is below slot_n.  Short mode runs only for rows of at most
// 512 words (S <= 32768), so source ids fit 15 bits.
using Tiny = uint32_t;
constexpr uint32_t TINY_MAX = 2;    // ids a tiny word holds
constexpr uint32_t CHUNK_IDS = 16;  // uint16 entries per 32-byte chunk of a slot

// Tiny word of a row of `total` bits; part = its first two ids (bits 0..14,
// 15..29) when total <= TINY_MAX.
__host__ __device__ __forceinline__ Tiny tiny_word(uint32_t total, uint32_t part) {
  return total == 0 ? 0u
         : total <= TINY_MAX ? (total << 30) | part
                             : (3u << 30) | (total < 0xFFFFu ? total : 0xFFFFu);
}
// Bit count of a row from its tiny word: exact up to TINY_MAX, else the
// saturated count.
__device__ __forceinline__ uint32_t tiny_count(Tiny t) {
  const uint32_t cls = t >> 30;
  return cls < 3 ? cls : (t & 0xFFFFu);
}

// Read-only tiny-word load that asks L2 to keep the line (evict-last).
__device__ __forceinline__ Tiny ld_keep(const Tiny *p) {
  uint64_t pol;
  asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol));
  Tiny r;
  asm("ld.global.nc.L2::cache_hint.b32 %0, [%1], %2;" : "=r"(r) : "l"(p), "l"(pol));
  return r;
}

// OR x into a union in global memory; it is read first: it is complete after a
// few rows and then costs no atomic.
__device__ __forceinline__ void add_union(uint4 *u, uint4 x) {
  const uint4 n = andnot4(x, __ldcg(u));
  unsigned *w = reinterpret_cast<unsigned *>(u);
  if (n.x) atomicOr(w, n.x);
  if (n.y) atomicOr(w + 1, n.y);
  if (n.z) atomicOr(w + 2, n.z);
  if (n.w) atomicOr(w + 3, n.w);
}

// ro, so, po: out-degrees of the layer's non-empty rows, of its short rows, and per bit
__device__ __forceinline__ void pull_counters(const PullArgs &a, unsigned long long nb, unsigned long long nv,
                                              unsigned long long ns, unsigned long long se, unsigned long long ro,
                                              unsigned long long so, unsigned long long po) {
  block_add(nb, &a.ctr->hop[a.h].new_bits);
  block_add(nv, &a.ctr->hop[a.h].active_vertices);
  if (a.tiny_out) {
    block_add(ns, &a.ctr->hop[a.h].short_rows);
    block_add(ro, &a.ctr->hop[a.h].row_out);
    block_add(so, &a.ctr->hop[a.h].short_out);
    block_add(po, &a.ctr->hop[a.h].pair_edges);
  }
  if (a.tiny_in) block_add(se, &a.ctr->hop[a.h].short_edges);
}

// ---------------------------------------------------------------------------
// Dense PULL.  L lanes hold a row (UPL uint4 per lane; L < 32 when the row is
// narrower than a warp), and a warp's G = 32 / L groups each own a target of
// their own: a group walks its target's in-list 8 or more entries a round with
// every row load in flight at once, so neither a reduction across groups nor a
// shuffle tree is paid per target.  What bounds it: row loads from L2 (rows of
// 256 bytes and more), else instructions and the latency of the chain offset ->
// neighbour -> flag -> row, which the groups of a warp overlap.
//
// Scheduling.  Warps take tasks of `tile` consecutive targets from a counter
// (in-degrees of R-MAT graphs follow the bits of the vertex id, so any fixed
// stride gives some warps a multiple of the mean work).  Targets above the
// heavy threshold are cut into pieces that come first
// in the same queue: a warp ORs a piece with all its groups, adds it to the
// target's union in HBM, and the warp that adds the last piece runs the
// epilogue.
//
// Early exit.  A row can only gain sources that some row of layer h-1 holds
// (their union, kept per layer by the PULL epilogues) and that the target has
// not visited: a target with nothing left to gain is skipped, and a list is
// left as soon as the row holds everything it could gain.  In the saturated
// hops of a small-world graph most targets stop within a few neighbours.
//
// Measured on GB300 against a warp per target at a fixed stride with a CTA per
// hub: R-MAT scale 16, 512 sources, hops 2 and 3 172 + 27 us -> 36 us each;
// 1M-vertex power law, 64 sources, hop 4 465 -> 151 us; R-MAT scale 20 both
// ways, 1,001 sources, hop 2 3.36 -> 0.55 ms; R-MAT scale 18, 3,000 sources, hops
// 3 to 5 1.38 ms -> 0.31, 0.20 and 0.17 ms; 4,096 sources on the 1M-vertex power
// law, hop 4 (no row saturates) 1.58 -> 1.43 ms at 10.7 TB/s of row loads.
constexpr uint32_t NONE = 0xffffffffu;
template <int L> constexpr int kChunk = L == 1 ? 8 : 32;

// Entries per piece and default heavy threshold: a piece of a narrow row is one
// or two rounds of a warp's groups, and the groups of a warp wait for its
// longest list, so narrow rows (many groups) cut earlier.
inline uint32_t piece_edges(int L) { return L <= 8 ? 512 : 256; }
inline uint32_t heavy_default(int L) { return L <= 8 ? 64 : 256; }
// Lists up to here are walked whole when the caller asks for it: four of them still
// number their entries in 32 bits.
constexpr uint32_t HEAVY_MAX = 1u << 28;

// Whether `p` holds on every lane of this lane's group.
template <int L> __device__ __forceinline__ bool group_all(bool p) {
  if (L == 1) return p;
  if (L == 32) return __all_sync(FULL, p);
  const unsigned gm = ((1u << (L & 31)) - 1u) << (threadIdx.x & 31 & ~(L - 1));
  return (__ballot_sync(FULL, p) & gm) == gm;
}

// Bits of uint4 q of a row that exist (sources below S).
__device__ __forceinline__ uint4 row_bits(uint32_t q, uint32_t S) {
  uint32_t w[4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const uint32_t b = q * 128 + i * 32;
    w[i] = b + 32 <= S ? 0xffffffffu : b < S ? (1u << (S - b)) - 1u : 0u;
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

__device__ __forceinline__ uint4 and4(uint4 a, uint4 b) {
  return make_uint4(a.x & b.x, a.y & b.y, a.z & b.z, a.w & b.w);
}

// Nothing left to gain: every bit of um is in vv or acc.
template <int L, int UPL>
__device__ __forceinline__ bool covered(const uint4 *s_um, uint32_t qn, const uint4 (&vv)[UPL], const uint4 (&acc)[UPL]) {
  const uint32_t gl = threadIdx.x & (L - 1);
  bool c = true;
#pragma unroll
  for (int k = 0; k < UPL; k++) {
    const uint32_t q = gl + k * L;
    if (q < qn) c = c && !nz4(andnot4(s_um[q], or4(vv[k], acc[k])));
  }
  return c;
}

// Whether vertex u has a row: its bit in shared memory (BITS) or its flag.
template <bool BITS> __device__ __forceinline__ bool has_row(const uint32_t *flag, uint32_t u) {
  return BITS ? flag[u >> 5] >> (u & 31) & 1u : __ldg(flag + u) != 0;
}

// OR the rows of list entries j, j + 1, ... (a group's rounds are `step` apart)
// below n into acc, until the row is covered.  Every lane of the warp calls it;
// a group with sat set only takes part in the votes.
template <int L, int UPL, bool BITS>
__device__ __forceinline__ void gather_list(const PullArgs &a, const uint4 *__restrict__ F, const uint32_t *flag,
                                            const uint4 *s_um, uint32_t qn, const uint32_t *__restrict__ adj,
                                            uint32_t n, uint32_t j, uint32_t step, const uint4 (&vv)[UPL],
                                            uint4 (&acc)[UPL], bool &sat) {
  const uint32_t lane = threadIdx.x & 31, gl = lane & (L - 1);
  if constexpr (L < 32) {
    constexpr int CH = kChunk<L>;  // entries per group and round, all requested at once
    constexpr int K = CH / L;         // ... per lane
    for (;;) {
      const bool more = !sat && j < n;
      if (!__any_sync(FULL, more)) break;
      uint32_t id[K];
#pragma unroll
      for (int k = 0; k < K; k++) {
        const uint32_t i = j + k * L + gl;
        id[k] = NONE;
        if (more && i < n) id[k] = __ldg(adj + i);
      }
      if (BITS && L <= 2) {  // rows of one sector: only the loads of the non-empty ones, in place
#pragma unroll
        for (int k = 0; k < K; k++)
          if (id[k] != NONE && !has_row<BITS>(flag, id[k])) id[k] = NONE;
      }
      if (!(BITS && L <= 2) && (BITS || flag)) {  // few rows of a round are non-empty: walk those
#pragma unroll
        for (int k = 0; k < K; k++)
          if (id[k] != NONE && !has_row<BITS>(flag, id[k])) id[k] = NONE;
#pragma unroll
        for (int k = 0; k < K; k++) {
          unsigned m = __ballot_sync(FULL, id[k] != NONE) >> (lane & ~(L - 1)) & ((1u << L) - 1u);
          while (__any_sync(FULL, m)) {
            uint4 x[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
              const uint32_t u = __shfl_sync(FULL, id[k], m ? __ffs(m) - 1 : 0, L);
              x[i] = make_uint4(0, 0, 0, 0);
              if (m && gl < qn) x[i] = __ldg(F + (size_t)u * a.Q + gl);
              m &= m - 1;
            }
#pragma unroll
            for (int i = 0; i < 4; i++) acc[0] = or4(acc[0], x[i]);
          }
        }
      } else {
#pragma unroll
        for (int i0 = 0; i0 < CH; i0 += 8) {
          if (i0 && !__any_sync(FULL, !sat && j + i0 < n)) break;
          uint4 x[8];
#pragma unroll
          for (int i = 0; i < 8; i++) {
            const uint32_t u = L == 1 ? id[(i0 + i) / L] : __shfl_sync(FULL, id[(i0 + i) / L], (i0 + i) % L, L);
            x[i] = make_uint4(0, 0, 0, 0);
            if (u != NONE && gl < qn) x[i] = __ldg(F + (size_t)u * a.Q + gl);
          }
#pragma unroll
          for (int i = 0; i < 8; i++) acc[0] = or4(acc[0], x[i]);
        }
      }
      j += step;
      const bool c = group_all<L>(covered<L, UPL>(s_um, qn, vv, acc));
      sat = sat || c;
    }
  } else {
    // The non-empty rows of 32 entries are numbered through shared memory, so that a
    // round of R rows is R addresses, loads and ORs without a search for the next bit,
    // a select and a test per row: 39 -> 21 warp instructions a list entry, which
    // bounds rows that come from L2 (40K vertices of 60 neighbours, 4,096 sources: 122 ->
    // 88 us a hop; the 1M-vertex power law's four hops 3.90 -> 3.63 ms).
    constexpr int R = UPL == 1 ? 8 : UPL == 2 ? 4 : 2;  // rows in flight
    __shared__ uint4 s_id[8][8];
    uint32_t *ids = reinterpret_cast<uint32_t *>(s_id[threadIdx.x >> 5]);
    for (; j < n && !sat; j += step) {
      uint32_t id = NONE;
      if (j + lane < n) id = __ldg(adj + j + lane);
      if ((BITS || flag) && id != NONE && !has_row<BITS>(flag, id)) id = NONE;
      const unsigned m = __ballot_sync(FULL, id != NONE);
      const int c = __popc(m);
      __syncwarp();  // every lane is past the last entries
      if (id != NONE) ids[__popc(m & lanemask_lt())] = id;
      __syncwarp();
      for (int t = 0; t < c; t += R) {
        uint32_t u[R];
#pragma unroll
        for (int k = 0; k < R; k++) u[k] = ids[t + k];  // R divides 32; those from c on are not used
        if (t + R <= c) {
#pragma unroll
          for (int i = 0; i < UPL; i++) {
            const uint32_t q = lane + i * 32;
            if (q < qn) {
              uint4 x[R];
#pragma unroll
              for (int k = 0; k < R; k++) x[k] = __ldg(F + (size_t)u[k] * a.Q + q);
#pragma unroll
              for (int k = 0; k < R; k++) acc[i] = or4(acc[i], x[k]);
            }
          }
        } else {
#pragma unroll
          for (int i = 0; i < UPL; i++) {
            const uint32_t q = lane + i * 32;
            uint4 x[R];
#pragma unroll
            for (int k = 0; k < R; k++) {
              x[k] = make_uint4(0, 0, 0, 0);
              if (t + k < c && q < qn) x[k] = __ldg(F + (size_t)u[k] * a.Q + q);
            }
#pragma unroll
            for (int k = 0; k < R; k++) acc[i] = or4(acc[i], x[k]);
          }
        }
        // whether the row is complete is asked every 8 rows: 60 instructions for a row of 8 uint4 a lane
        if ((t + R) % 8 == 0 && (t + R < c || j + step < n) && group_all<32>(covered<L, UPL>(s_um, qn, vv, acc))) {
          sat = true;
          break;
        }
      }
    }
  }
}

// Group form of write_short for every group of the warp at once: the tiny
// word and slot of the group's row x (valid: the group has a target, nz: its
// row is not empty), c the lane's bit count.  Returns whether the row is short.
template <int L, int UPL, int NW>
__device__ __forceinline__ bool write_short_group(const PullArgs &a, uint32_t v, bool valid, bool nz,
                                                  const uint4 (&x)[UPL], uint32_t qn, uint32_t c,
                                                  unsigned long long &ns) {
  constexpr int G = 32 / L, SQ = G * 2 > 8 ? G * 2 : 8;
  // slots of up to 64 entries where a warp holds one row (L == 32), of 16 below
  __shared__ uint4 s_stage[NW][SQ];
  const uint32_t lane = threadIdx.x & 31, gl = lane & (L - 1), g = lane / L;
  uint32_t incl = c;
#pragma unroll
  for (int o = 1; o < L; o <<= 1) {
    const uint32_t y = __shfl_up_sync(FULL, incl, o, L);
    if (gl >= (uint32_t)o) incl += y;
  }
  const uint32_t total = L == 1 ? c : __shfl_sync(FULL, incl, L - 1, L);
  const bool fits = valid && nz && total < a.slot_n;
  uint4 *stage4 = &s_stage[threadIdx.x >> 5][L == 32 ? 0 : g * 2];
  uint16_t *stage = reinterpret_cast<uint16_t *>(stage4);
  uint4 *slot = reinterpret_cast<uint4 *>(a.slot_out + (size_t)v * a.slot_n);
  if (fits && c) {
    uint32_t pos = 1 + incl - c;
#pragma unroll
    for (int k = 0; k < UPL; k++) {
      const uint32_t q = gl + k * L;
      if (q < qn) {
        const uint32_t w[4] = {x[k].x, x[k].y, x[k].z, x[k].w};
#pragma unroll
        for (int wi = 0; wi < 4; wi++) {
          uint32_t bits = w[wi];
          while (bits) {
            stage[pos++] = (uint16_t)(q * 128 + wi * 32 + __ffs(bits) - 1);
            bits &= bits - 1;
          }
        }
      }
    }
  }
  if (fits && gl == 0) stage[0] = (uint16_t)total;
  __syncwarp();
  if (fits)
    for (uint32_t i = gl; i < a.slot_n / 8; i += L) slot[i] = stage4[i];
  if (valid && gl == 0) {
    if (!nz) {
      a.tiny_out[v] = 0;
      a.slot_out[(size_t)v * a.slot_n] = 0;
    } else if (!fits) {  // a long row: its count alone
      a.tiny_out[v] = tiny_word(total, 0);
      a.slot_out[(size_t)v * a.slot_n] = (uint16_t)(total < 0xFFFFu ? total : 0xFFFFu);
    } else {
      a.tiny_out[v] = tiny_word(total, total <= TINY_MAX ? stage[1] | (total > 1 ? (uint32_t)stage[2] << 15 : 0u) : 0u);
      ns += 1ull + (total <= TINY_MAX ? 1ull << 32 : 0ull);
    }
  }
  __syncwarp();  // the staging slots are free for the warp's next round
  return fits;
}

// Epilogue of a round: every group's target v (valid per group), its ORed rows
// acc and visited words vv: visited update, accumulator OR, layer union,
// next-layer row (with its tiny word and slot), flag, counters.
template <int L, int UPL, int NW>
__device__ __forceinline__ void group_epilogue(const PullArgs &a, uint32_t v, bool valid, uint32_t q0, uint32_t qn,
                                               const uint4 *s_um, uint4 *s_un, const uint4 (&vv)[UPL], uint4 (&acc)[UPL],
                                               unsigned long long &nb, unsigned long long &nv, unsigned long long &ns,
                                               unsigned long long &ro, unsigned long long &so,
                                               unsigned long long &po) {
  const uint32_t lane = threadIdx.x & 31, gl = lane & (L - 1);
  bool any = false;
  uint32_t bits = 0;
#pragma unroll
  for (int k = 0; k < UPL; k++) {
    const uint32_t q = gl + k * L;
    uint4 x = make_uint4(0, 0, 0, 0);
    if (valid && q < qn) {
      x = and4(andnot4(acc[k], vv[k]), s_um[q]);
      if (nz4(x)) {
        const size_t idx = (size_t)v * a.Q + q0 + q;
        any = true;
        bits += popc4(x);
        if (a.shortest) a.vis[idx] = or4(vv[k], x);
        if (a.acc_on) {
          const uint4 o = a.acc[idx];
          if (nz4(andnot4(x, o))) a.acc[idx] = or4(o, x);
        }
        if (!a.last) {
          const uint4 n = andnot4(x, s_un[q]);
          unsigned *w = reinterpret_cast<unsigned *>(s_un + q);
          if (n.x) atomicOr(w, n.x);
          if (n.y) atomicOr(w + 1, n.y);
          if (n.z) atomicOr(w + 2, n.z);
          if (n.w) atomicOr(w + 3, n.w);
        }
      }
    }
    acc[k] = x;
  }
  nb += bits;
  const bool rownz = !group_all<L>(!any);
  if (valid && gl == 0 && rownz && (a.res_vis || a.acc_on)) a.resflag[v] = 1;
  if (a.multislice) {
    if (valid && rownz) {
#pragma unroll
      for (int k = 0; k < UPL; k++) {
        const uint32_t q = gl + k * L;
        if (q < qn && nz4(acc[k])) a.N[(size_t)v * a.Q + q0 + q] = acc[k];
      }
      if (gl == 0 && atomicOr(&a.flagN[v], 1u) == 0) nv++;
    }
    return;
  }
  const uint32_t oldf = valid ? a.flagN[v] : 0u;  // 1: the buffer row holds an older layer's bits
  if (a.last) {
    // layer k_max is not kept: clear the rows an earlier layer left in this
    // buffer, so the next run finds it clean (a flag-2 row is zero already)
    if (oldf == 1) {
#pragma unroll
      for (int k = 0; k < UPL; k++) {
        const uint32_t q = gl + k * L;
        if (q < qn) a.N[(size_t)v * a.Q + q0 + q] = make_uint4(0, 0, 0, 0);
      }
    }
    __syncwarp();  // every lane of a group read its flag
    if (valid && gl == 0) {
      if (oldf) a.flagN[v] = 0;
      nv += rownz;
    }
    return;
  }
  bool virt = false;  // the row is left in its slot only (flag 2)
  if (!(NW > 8 && L < 16) && a.tiny_out) {
    const bool fits = write_short_group<L, UPL, NW>(a, v, valid, rownz, acc, qn, bits, ns);
    virt = fits && a.virt_out;
    if (valid && rownz && (bits || gl == 0)) {
      const unsigned long long d = out_degree(a.out, v);
      po += d * bits;
      if (gl == 0) ro += d;
      if (gl == 0 && fits) so += d;
    }
  }
  if (valid && ((rownz && !virt) || oldf == 1)) {
#pragma unroll
    for (int k = 0; k < UPL; k++) {
      const uint32_t q = gl + k * L;
      if (q < qn) a.N[(size_t)v * a.Q + q0 + q] = virt ? make_uint4(0, 0, 0, 0) : acc[k];
    }
  }
  __syncwarp();
  if (valid && gl == 0) {
    const uint32_t nf = rownz ? (virt ? 2u : 1u) : 0u;
    if (nf != oldf) a.flagN[v] = nf;
    nv += rownz;
  }
}

// BITS: the flags of layer h-1 as bits in shared memory, one block of 32 warps an SM.
// A flag in global memory costs an L1 tag and mostly an L2 sector per list entry (5 ps
// on the whole chip, as much as a row of one uint4); its bit costs a shared-memory word.
// 64 sources on the 1M-vertex power law, hop 3 (5% of the rows active) 149 -> 94 us;
// 1,001 sources both ways on R-MAT 20, hops 2 to 5 2.25 -> 2.06 ms; 2,048 sources on the
// power law, two hops 1.20 -> 1.09 ms.
template <int L, int UPL, bool BITS>
__global__ void __launch_bounds__(BITS ? 1024 : 256, BITS ? 1 : UPL == 1 ? 4 : UPL == 2 ? 3 : 2)
    k_pull(PullArgs a) {
  vs::grid_wait();
  HopCtr &hc = a.ctr->hop[a.h];
  if (hc.strategy != ST_PULL || hc.short_pull || (hc.bits != 0) != BITS) return;
  constexpr int NW = BITS ? 32 : 8;  // warps
  extern __shared__ uint4 s_bits[];
  if (BITS)
    for (uint32_t i = threadIdx.x; i < (a.V + 127) / 128; i += blockDim.x)
      s_bits[i] = __ldg(reinterpret_cast<const uint4 *>(a.bits) + i);
  constexpr uint32_t G = 32 / L, CH = kChunk<L>;
  __shared__ uint4 s_um[L * UPL];  // what a row can gain: the union of layer h-1, rows still growing
  __shared__ uint4 s_un[L * UPL];  // union of the rows this block wrote
  const uint32_t lane = threadIdx.x & 31, g = lane / L, gl = lane & (L - 1);
  const uint32_t q0 = blockIdx.y * a.qslice, qn = min(a.qslice, a.Q - q0);
  const HopCtr &pc = a.ctr->hop[a.h - 1];
  for (uint32_t q = threadIdx.x; q < qn; q += blockDim.x) {
    uint4 m = pc.strategy == ST_PULL ? a.Uin[q0 + q] : row_bits(q0 + q, a.S);
    if (a.hmask) m = and4(m, a.hmask[q0 + q]);
    s_um[q] = m;
    s_un[q] = make_uint4(0, 0, 0, 0);
  }
  __syncthreads();
  // a row of one sector is loaded as fast as its flag, and a nearly full layer has few
  // rows to skip.  On a graph below the bits' size a hop is bound by its chains of loads:
  // rows of up to four uint4 come without the flag before them, eight at a time (R-MAT of
  // 4K to 64K vertices, 300 to 500 sources: 6 to 20% of a run, power laws 1 to 12%; wider
  // rows lose up to 4% at eight uint4 and 13% at sixteen)
  const bool useflag = a.Q > 2 && pc.active_vertices * 10 < 9ull * a.V && !(L <= 4 && a.V < BITS_MIN_V);
  const uint32_t *flag = BITS ? reinterpret_cast<const uint32_t *>(s_bits) : useflag ? a.flagF : nullptr;
  const uint4 *F = a.F + q0;
  const bool known = a.res_vis && a.Q >= 8;  // resflag 0: the visited row is zero, without reading it
  // rows are often complete only once a good part of all bits is visited; before
  // that the visited words arrive while the first neighbours are fetched
  unsigned long long seen = 0;
  if (a.shortest)
    for (int i = 0; i < a.h; i++) seen += a.ctr->hop[i].new_bits;
  const bool precheck = seen > (unsigned long long)a.V * a.S / 8;
  const uint32_t ntasks = a.npieces + (a.V + a.tile - 1) / a.tile;
  unsigned long long nb = 0, nv = 0, ns = 0, ro = 0, so = 0, po = 0;
  auto fetch = [&]() {
    uint32_t t = 0;
    if (lane == 0) t = atomicAdd(a.queue + blockIdx.y, 1u);
    return t;  // lane 0's; broadcast when used
  };
  auto visited = [&](uint32_t v, bool valid, uint4(&vv)[UPL]) {
    const bool look = valid && a.shortest && (!known || a.resflag[v]);
#pragma unroll
    for (int k = 0; k < UPL; k++) {
      vv[k] = make_uint4(0, 0, 0, 0);
      const uint32_t q = gl + k * L;
      if (look && q < qn) vv[k] = a.vis[(size_t)v * a.Q + q0 + q];
    }
  };
  uint32_t task = __shfl_sync(FULL, fetch(), 0);
  while (task < ntasks) {
    const uint32_t nexttask = fetch();  // in flight during this task
    uint4 vv[UPL], acc[UPL];
    if (task < a.npieces) {
      const uint4 pc4 = __ldg(a.pieces + task);
      const uint32_t v = pc4.x, np = pc4.y == NONE ? 1u : a.heavy_np[pc4.y];
      uint4 *sum = a.heavy_rows + (np > 1 ? (size_t)pc4.y * a.Q + q0 : 0);
      visited(v, true, vv);
      uint4 cov[UPL];
#pragma unroll
      for (int k = 0; k < UPL; k++) {
        acc[k] = make_uint4(0, 0, 0, 0);
        cov[k] = vv[k];
        const uint32_t q = gl + k * L;
        if (np > 1 && q < qn) cov[k] = or4(cov[k], __ldcg(sum + q));  // what other pieces found already
      }
      bool sat = group_all<L>(covered<L, UPL>(s_um, qn, cov, acc));
      const int64_t beg = a.in.off[pc4.z][v], end = a.in.off[pc4.z][v + 1];
      const uint32_t n = (uint32_t)min((int64_t)pc4.w + a.piece_edges, end - beg);
      gather_list<L, UPL, BITS>(a, F, flag, s_um, qn, a.in.adj[pc4.z] + beg, n, pc4.w + (L < 32 ? g * CH : 0),
                          L < 32 ? G * CH : 32, cov, acc, sat);
#pragma unroll
      for (int o = L; o < 32; o <<= 1)
#pragma unroll
        for (int k = 0; k < UPL; k++) acc[k] = or4(acc[k], shfl_xor4(acc[k], o));
      bool mine = true;
      if (np > 1) {
        if (g == 0) {
#pragma unroll
          for (int k = 0; k < UPL; k++) {
            const uint32_t q = gl + k * L;
            if (q < qn) add_union(sum + q, acc[k]);
          }
          __threadfence();
        }
        __syncwarp();
        uint32_t left = 0;
        uint32_t *cnt = a.heavy_left + (size_t)pc4.y * gridDim.y + blockIdx.y;
        if (lane == 0) left = atomicSub(cnt, 1u);
        left = __shfl_sync(FULL, left, 0);
        mine = left == 1;
        if (mine) {  // the last piece: the whole union, and both left as they were found
          __threadfence();
#pragma unroll
          for (int k = 0; k < UPL; k++) {
            const uint32_t q = gl + k * L;
            acc[k] = make_uint4(0, 0, 0, 0);
            if (q < qn) acc[k] = __ldcg(sum + q);
          }
          __syncwarp();
          if (g == 0) {
#pragma unroll
            for (int k = 0; k < UPL; k++) {
              const uint32_t q = gl + k * L;
              if (q < qn) sum[q] = make_uint4(0, 0, 0, 0);
            }
          }
          if (lane == 0) *cnt = np;
        }
      }
      if (mine) group_epilogue<L, UPL, NW>(a, v, g == 0, q0, qn, s_um, s_un, vv, acc, nb, nv, ns, ro, so, po);
    } else {
      // the tile's list starts at once: lane i holds those of target v0 + i (a tile of
      // L > 1 has at most 16 targets, so lane i + 1 holds the end too)
      const uint32_t v0 = (task - a.npieces) * a.tile;
      int64_t off[2] = {0, 0}, oend[2] = {0, 0};
      _Pragma("unroll") for (int l = 0; l < 2; l++) if (l < a.in.n) {
        off[l] = __ldg(a.in.off[l] + min(v0 + lane, a.V));
        if (L == 1) oend[l] = __ldg(a.in.off[l] + min(v0 + lane + 1, a.V));
      }
      for (uint32_t r = 0; r < a.tile && v0 + r < a.V; r += G) {
        const uint32_t v = v0 + r + g;
        bool valid = v < a.V;
        int64_t beg[2] = {0, 0};
        uint32_t n[2] = {0, 0};
        uint64_t d = 0;
        _Pragma("unroll") for (int l = 0; l < 2; l++) if (l < a.in.n) {
          beg[l] = L == 1 ? off[l] : __shfl_sync(FULL, off[l], r + g);
          n[l] = (uint32_t)((L == 1 ? oend[l] : __shfl_sync(FULL, off[l], r + g + 1)) - beg[l]);
          d += n[l];
        }
        if (a.heavy_threshold && d > a.heavy_threshold) valid = false;  // comes in pieces
        visited(v, valid, vv);
#pragma unroll
        for (int k = 0; k < UPL; k++) acc[k] = make_uint4(0, 0, 0, 0);
        bool sat = !valid;
        if (precheck) {
          const bool c = group_all<L>(covered<L, UPL>(s_um, qn, vv, acc));
          sat = sat || c;
        }
        _Pragma("unroll") for (int l = 0; l < 2; l++) if (l < a.in.n)
          gather_list<L, UPL, BITS>(a, F, flag, s_um, qn, a.in.adj[l] + beg[l], n[l], 0, L < 32 ? CH : 32, vv, acc, sat);
        group_epilogue<L, UPL, NW>(a, v, valid, q0, qn, s_um, s_un, vv, acc, nb, nv, ns, ro, so, po);
      }
    }
    task = __shfl_sync(FULL, nexttask, 0);
  }
  pull_counters(a, nb, nv, ns, 0, ro, so, po);
  __syncthreads();
  if (!a.last)
    for (uint32_t q = threadIdx.x; q < qn; q += blockDim.x) add_union(a.Uout + q0 + q, s_un[q]);
}

// ---------------------------------------------------------------------------
// Short-mode PULL (one slice).  A warp takes T consecutive targets and keeps
// their rows as bitmaps in shared memory.  Their in-lists lie end to end in the
// CSR and are read as one range, 32 edges at a time whatever the degrees, a lane
// per edge, the loads of several such rounds in flight at once:
//   words  a lane per edge ORs its word's ids; where they are also appended to lists
//          (LIST), and most edges come from empty rows, they are queued and taken 32 at
//          a time, a full warp whatever target they belong to;
//   slots  a lane per edge ORs its slot's ids.
// In-neighbours with 16 ids or more are put aside: those with a slot are done by
// all lanes, an id each, the others are rows gathered whole.
//
// Three ways to finish a tile:
//   LIST  (word hops) the bitmaps start as the visited rows, so the atomic's old
//         word tells a new id, which is appended to the target's list at once: the
//         list is the slot of the next layer and no row is searched for bits.
//         Long rows, and targets that got a whole row, are done from the bitmap.
//   LAST  nothing follows the layer: the bitmaps start as the visited rows and
//         are written back; popcounts before and after give the new bits.
//   GEN   any other hop (slots, accumulator, kept layer, long new rows): the bitmaps
//         start empty and finish_row does every touched target.
//
// What bounds it: instructions and latency (2M-vertex power law, 28 edges a target,
// 2,048 sources: 200 warp instructions a target where lists are kept, 490 where every
// target was searched, 0.75 issued a cycle and scheduler), not DRAM.  So no call in a kernel's loops (around one, 40 registers went to local
// memory that L1 could not hold: 2.2 times slower), words and slots in kernels of
// their own (together they spill), four targets a tile (eight halve what is left of
// L1: 7.85 -> 12.2 ms on the 10M-vertex slot hop).  Against a warp per target with
// its row in registers, 4,096 sources: 1M-vertex power law, the hop after SPARSE 545
// (a dense hop; short mode did not pay) -> 345 us; backward lists, 2,048 sources 645 +
// a CTA per hub 409 -> 755 us; 10M vertices, third hop 5.56 -> 5.0 ms, last hop 7.88
// -> 7.7 ms.
enum { SH_LIST = 0, SH_LAST = 1, SH_GEN = 2 };
constexpr int SH_WARPS = 8;

// Shared memory of a block, in uint4: the union of the rows it wrote [Q], the
// rows that may still grow [Q] (with row limits), then per warp, from wb on:
// bitmap rows [T][Q], lists of slot_n entries (entry 0: the count) [T] from
// sh_list, counts of the lists and queue of ids from sh_queue, in-neighbours put
// aside (id, target | count << 8) from sh_aside.
extern __shared__ uint4 s_short[];

// A slot's first 32 bytes (32-byte aligned) in one load that leaves L1 to the lists.
__device__ __forceinline__ void ld_slot(const uint4 *p, uint4 &x, uint4 &y) {
  asm("ld.global.nc.L1::no_allocate.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(x.x), "=r"(x.y), "=r"(x.z), "=r"(x.w), "=r"(y.x), "=r"(y.y), "=r"(y.z), "=r"(y.w)
      : "l"(p));
}

// A lane's id into a target's bitmap, the old word unused.
__device__ __forceinline__ void or_id(uint32_t *row, uint32_t id) { atomicOr(row + (id >> 5), 1u << (id & 31)); }

// Whether an id's row may still grow.
__device__ __forceinline__ bool may_grow(const PullArgs &a, uint32_t id) {
  return !a.hmask || (reinterpret_cast<const uint32_t *>(s_short + a.Q)[id >> 5] >> (id & 31) & 1u);
}

// Every lane with act ORs its id into target own's bitmap; LIST: new ids are
// appended to the targets' lists.
template <int MODE>
__device__ __forceinline__ void put_ids(const PullArgs &a, uint32_t wb, bool act, uint32_t own, uint32_t id) {
  act = act && may_grow(a, id);
  const uint32_t w = id >> 5, bit = 1u << (id & 31);
  uint32_t *row = reinterpret_cast<uint32_t *>(s_short + wb + own * a.Q);
  if (MODE != SH_LIST) {
    if (act) atomicOr(row + w, bit);
    return;
  }
  const bool fresh = act && !(atomicOr(row + w, bit) & bit);
  const unsigned m = __ballot_sync(FULL, fresh);
  if (!m) return;
  const unsigned peers = __match_any_sync(FULL, fresh ? own : 32u);
  uint32_t *cnt = reinterpret_cast<uint32_t *>(s_short + wb + a.sh_queue) + own;
  if (fresh) {
    const uint32_t base = *cnt, at = 1 + base + __popc(peers & lanemask_lt());
    if (at < a.slot_n) reinterpret_cast<uint16_t *>(s_short + wb + a.sh_list)[own * a.slot_n + at] = (uint16_t)id;
    uint32_t *un = reinterpret_cast<uint32_t *>(s_short) + w;
    if (!(*un & bit)) atomicOr(un, bit);
  }
  __syncwarp();
  if (fresh && (peers & lanemask_lt()) == 0) *cnt += __popc(peers);
  __syncwarp();
}

// The n in-neighbours put aside, two at a time: rows with a slot an id per lane,
// others whole.  Returns the targets that got a whole row.
template <int MODE> __device__ __forceinline__ unsigned do_aside(const PullArgs &a, uint32_t wb, uint32_t naside) {
  const uint32_t lane = threadIdx.x & 31;
  const uint2 *aside = reinterpret_cast<const uint2 *>(s_short + wb + a.sh_aside);
  const uint16_t *slots = reinterpret_cast<const uint16_t *>(a.slot_in);
  unsigned whole = 0;
  for (uint32_t k = 0; k < naside; k += 2) {
    uint2 e[2];
    uint32_t id[2];
#pragma unroll
    for (int i = 0; i < 2; i++) {
      e[i] = k + i < naside ? aside[k + i] : make_uint2(0, 0);
      const uint32_t c = e[i].y >> 8;
      id[i] = c < a.slot_n && lane < c ? __ldg(slots + (size_t)e[i].x * a.slot_n + 1 + lane) : 0u;
    }
    if ((e[0].y >> 8) >= a.slot_n || (e[1].y >> 8) >= a.slot_n) {
      for (uint32_t q = lane; q < a.Q; q += 32) {
        uint4 x[2];
#pragma unroll
        for (int i = 0; i < 2; i++) {
          x[i] = make_uint4(0, 0, 0, 0);
          if ((e[i].y >> 8) >= a.slot_n) x[i] = __ldg(a.F + (size_t)e[i].x * a.Q + q);
        }
#pragma unroll
        for (int i = 0; i < 2; i++)
          if ((e[i].y >> 8) >= a.slot_n) {
            uint4 *p = s_short + wb + (e[i].y & 255u) * a.Q + q;
            if (a.hmask) x[i] = and4(x[i], s_short[a.Q + q]);
            *p = or4(*p, x[i]);
          }
      }
      __syncwarp();
    }
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const uint32_t c = e[i].y >> 8, own = e[i].y & 255u;
      if (c >= a.slot_n) {
        whole |= 1u << own;
      } else {
        for (uint32_t i0 = 0; i0 < c; i0 += 32) {
          const bool act = i0 + lane < c;
          const uint32_t x = !i0 ? id[i] : act ? __ldg(slots + (size_t)e[i].x * a.slot_n + 1 + i0 + lane) : 0u;
          put_ids<MODE>(a, wb, act, own, x);
        }
      }
    }
    __syncwarp();  // ids are in before the next pair's whole rows are added word by word
  }
  return whole;
}

// The new bits of the T targets from v0 on that are in fm, from their bitmap rows (raw
// unions, or unions and visited bits): row & ~visited, left in the bitmap; visited,
// accumulator, union.  The targets' visited and accumulator cells are in flight at
// once: one target after the other cost a chain of three misses each (4,096 sources on
// the 10M-vertex power law, a hop into an accumulator, 8.4 -> 7.7 ms).  Lane t gets
// target t's number of new bits.
template <int T>
__device__ __forceinline__ uint32_t new_bits(const PullArgs &a, uint32_t wb, unsigned fm, uint32_t v0) {
  uint4 *rows = s_short + wb, *s_un = s_short;
  const uint4 *hm = a.hmask ? s_short + a.Q : nullptr;
  const uint32_t lane = threadIdx.x & 31;
  __syncwarp();
  uint32_t bits[T];
#pragma unroll
  for (int t = 0; t < T; t++) bits[t] = 0;
  for (uint32_t q = lane; q < a.Q; q += 32) {
    uint4 x[T], y[T];
#pragma unroll
    for (int t = 0; t < T; t++) {
      x[t] = fm >> t & 1u ? rows[t * a.Q + q] : make_uint4(0, 0, 0, 0);
      if (hm) x[t] = and4(x[t], hm[q]);
    }
    if (a.shortest) {
#pragma unroll
      for (int t = 0; t < T; t++) y[t] = nz4(x[t]) ? a.vis[(size_t)(v0 + t) * a.Q + q] : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int t = 0; t < T; t++) {
        x[t] = andnot4(x[t], y[t]);
        if (nz4(x[t])) a.vis[(size_t)(v0 + t) * a.Q + q] = or4(y[t], x[t]);
      }
    }
    if (a.acc_on) {
#pragma unroll
      for (int t = 0; t < T; t++) y[t] = nz4(x[t]) ? a.acc[(size_t)(v0 + t) * a.Q + q] : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int t = 0; t < T; t++)
        if (nz4(andnot4(x[t], y[t]))) a.acc[(size_t)(v0 + t) * a.Q + q] = or4(y[t], x[t]);
    }
    uint4 u = x[0];
#pragma unroll
    for (int t = 1; t < T; t++) u = or4(u, x[t]);
    if (!a.last) {
      const uint4 n = andnot4(u, s_un[q]);
      unsigned *w = reinterpret_cast<unsigned *>(s_un + q);
      if (n.x) atomicOr(w, n.x);
      if (n.y) atomicOr(w + 1, n.y);
      if (n.z) atomicOr(w + 2, n.z);
      if (n.w) atomicOr(w + 3, n.w);
    }
#pragma unroll
    for (int t = 0; t < T; t++)
      if (fm >> t & 1u) {
        rows[t * a.Q + q] = x[t];
        bits[t] += popc4(x[t]);
      }
  }
  uint32_t total = 0;
#pragma unroll
  for (int t = 0; t < T; t++) {
    const uint32_t n = __reduce_add_sync(FULL, bits[t]);
    if (lane == t) total = n;
  }
  return total;
}

// What follows from target t's new bits (in its bitmap row, `total` of them): next-layer
// row, word, slot, flag (oldf before).
__device__ __forceinline__ void finish_row(const PullArgs &a, uint32_t wb, uint32_t t, uint32_t v, uint32_t total,
                                           uint32_t oldf) {
  uint4 *row = s_short + wb + t * a.Q;
  uint16_t *list = reinterpret_cast<uint16_t *>(s_short + wb + a.sh_list) + t * a.slot_n;
  const uint32_t lane = threadIdx.x & 31;
  if (lane == 0 && total && (a.res_vis || a.acc_on)) a.resflag[v] = 1;
  if (a.last) {  // layer k_max is not kept: leave the buffer row and its flag clean
    if (oldf == 1)
      for (uint32_t q = lane; q < a.Q; q += 32) a.N[(size_t)v * a.Q + q] = make_uint4(0, 0, 0, 0);
    if (lane == 0 && oldf) a.flagN[v] = 0;
    return;
  }
  bool virt = false;
  if (a.tiny_out) {
    uint4 *slot = reinterpret_cast<uint4 *>(a.slot_out + (size_t)v * a.slot_n);
    if (total && total < a.slot_n) {
      uint32_t pos = 1;
      for (uint32_t q0 = 0; q0 < a.Q; q0 += 32) {
        const uint32_t q = q0 + lane;
        const uint4 x = q < a.Q ? row[q] : make_uint4(0, 0, 0, 0);
        const uint32_t n = popc4(x);
        uint32_t incl = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t y = __shfl_up_sync(FULL, incl, o);
          if (lane >= (uint32_t)o) incl += y;
        }
        uint32_t at = pos + incl - n;
        const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int wi = 0; wi < 4; wi++)
          for (uint32_t b = w[wi]; b; b &= b - 1) list[at++] = (uint16_t)(q * 128 + wi * 32 + __ffs(b) - 1);
        pos += __shfl_sync(FULL, incl, 31);
      }
      if (lane == 0) list[0] = (uint16_t)total;
      __syncwarp();
      if (lane < a.slot_n / 8) slot[lane] = reinterpret_cast<const uint4 *>(list)[lane];
      if (lane == 0)
        a.tiny_out[v] = tiny_word(total, total <= TINY_MAX ? list[1] | (total > 1 ? (uint32_t)list[2] << 15 : 0u) : 0u);
      virt = a.virt_out;
      __syncwarp();
    } else if (lane == 0) {
      a.tiny_out[v] = tiny_word(total, 0);
      a.slot_out[(size_t)v * a.slot_n] = (uint16_t)(total < 0xFFFFu ? total : 0xFFFFu);
    }
  }
  if ((total && !virt) || oldf == 1)
    for (uint32_t q = lane; q < a.Q; q += 32)
      a.N[(size_t)v * a.Q + q] = virt ? make_uint4(0, 0, 0, 0) : row[q];
  if (lane == 0) {
    const uint32_t nf = total ? (virt ? 2u : 1u) : 0u;
    if (nf != oldf) a.flagN[v] = nf;
  }
}

// What a warp carries over the edges of its tile.
struct ShortEdges {
  uint32_t wb, nq, naside, se;  // shared memory; ids queued, in-neighbours put aside, edges served (this lane)
  unsigned whole, touched;      // targets that got a whole row; any id
};

constexpr int SLOT_LANES = 4;                       // slots of 32 and more ids among 32 edges worth reading in place
constexpr uint32_t SH_GROUP = 2;                    // word hops: 32-edge items per round
constexpr uint32_t SH_IDS = 32 + SH_GROUP * 64;     // queued ids at most
constexpr uint32_t SH_ASIDE = 32 + SH_GROUP * 32;   // in-neighbours put aside at most

// Lanes with act queue an id for their target.
__device__ __forceinline__ void queue_id(const PullArgs &a, ShortEdges &s, bool act, uint32_t own, uint32_t id) {
  const unsigned m = __ballot_sync(FULL, act);
  uint32_t *q = reinterpret_cast<uint32_t *>(s_short + s.wb + a.sh_queue) + 8;  // past the counts
  if (act) q[s.nq + __popc(m & lanemask_lt())] = id | own << 16;
  s.nq += __popc(m);
}

__device__ __forceinline__ void put_aside(const PullArgs &a, ShortEdges &s, bool act, uint32_t own, uint32_t u,
                                          uint32_t n) {
  const unsigned m = __ballot_sync(FULL, act);
  if (!m) return;
  if (act)
    reinterpret_cast<uint2 *>(s_short + s.wb + a.sh_aside)[s.naside + __popc(m & lanemask_lt())] =
        make_uint2(u, own | n << 8);
  s.naside += __popc(m);
}

// OR the queued ids into the bitmaps, 32 at a time; all: the last ones too.
template <int MODE> __device__ __forceinline__ void drain(const PullArgs &a, ShortEdges &s, bool all) {
  const uint32_t lane = threadIdx.x & 31;
  if (s.nq >= 32 || (all && s.nq)) {
    uint32_t *q = reinterpret_cast<uint32_t *>(s_short + s.wb + a.sh_queue) + 8;
    __syncwarp();
    uint32_t at = 0;
    for (; at + 32 <= s.nq || (all && at < s.nq); at += 32) {
      const bool act = at + lane < s.nq;
      const uint32_t e = act ? q[at + lane] : 0u;
      put_ids<MODE>(a, s.wb, act, e >> 16, e & 0x7FFFu);
    }
    const uint32_t left = at < s.nq ? s.nq - at : 0u, e = lane < left ? q[at + lane] : 0u;
    __syncwarp();
    if (lane < left) q[lane] = e;
    s.nq = left;
  }
  if (s.naside >= 32 || (all && s.naside)) {
    __syncwarp();
    s.whole |= do_aside<MODE>(a, s.wb, s.naside);
    s.naside = 0;
    __syncwarp();
  }
}

// ids 1..n of a slot's first 32 bytes into a target's bitmap.
__device__ __forceinline__ void or_chunk(const PullArgs &a, uint32_t *row, uint32_t n, uint32_t mx, const uint4 x,
                                         const uint4 y) {
  const uint32_t w[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
#pragma unroll
  for (uint32_t i = 1; i < CHUNK_IDS; i++) {
    if (i > mx) break;
    const uint32_t id = i & 1 ? w[i >> 1] >> 16 : w[i >> 1] & 0xFFFFu;
    if (i <= n && may_grow(a, id)) or_id(row, id);
  }
}

// The same for the lanes with n ids in vertex u's slot, loaded here.
__device__ __forceinline__ void or_slot(const PullArgs &a, uint32_t *row, uint32_t n, uint32_t u) {
  uint4 x = make_uint4(0, 0, 0, 0), y = x;
  if (n) ld_slot(a.slot_in + (size_t)u * (a.slot_n / 8), x, y);
  or_chunk(a, row, n, __reduce_max_sync(FULL, n), x, y);
}

// 32 edges of a word hop: u the neighbour (NONE: no edge), t its word, own the target.
template <int MODE>
__device__ __forceinline__ void word_edges(const PullArgs &a, ShortEdges &s, uint32_t own, uint32_t u, Tiny t) {
  if (!__any_sync(FULL, t)) return;
  const uint32_t cls = t >> 30;
  if (MODE == SH_GEN) s.touched |= __reduce_or_sync(FULL, t ? 1u << own : 0u);
  const uint32_t id0 = t & 0x7FFFu, id1 = t >> 15 & 0x7FFFu;
  const bool one = cls == 1 || cls == 2;
  uint32_t *row = reinterpret_cast<uint32_t *>(s_short + s.wb + own * a.Q);
  if (MODE == SH_LIST)
    queue_id(a, s, one, own, id0);
  else if (one && may_grow(a, id0))  // no list to append to: into the bitmap at once
    or_id(row, id0);
  uint32_t n = cls;
  if (__any_sync(FULL, cls > 1)) {
    if (MODE == SH_LIST)
      queue_id(a, s, cls == 2, own, id1);
    else if (cls == 2 && may_grow(a, id1))
      or_id(row, id1);
    if (cls == 3) n = t & 0xFFFFu;
    // 3 to 15 ids: each lane its own slot where no list grows, else put aside, an id per
    // lane of the warp (put aside always, layers of 3 to 5 ids a row took 1.6 times as long)
    const bool held = MODE != SH_LIST && cls == 3 && n < CHUNK_IDS;
    put_aside(a, s, cls == 3 && !held, own, u, n);
    if (MODE != SH_LIST && __any_sync(FULL, held)) or_slot(a, row, held ? n : 0u, u);
  }
  s.se += n && n < a.slot_n;
}

// 32 edges of a slot hop: u the neighbour, its slot's first 32 bytes.
template <int MODE, bool WIDE>
__device__ __forceinline__ void slot_edges(const PullArgs &a, ShortEdges &s, uint32_t own, uint32_t u,
                                           const uint4 first, const uint4 second) {
  uint32_t n = first.x & 0xFFFFu;
  if (!__any_sync(FULL, n)) return;
  if (MODE == SH_GEN) s.touched |= __reduce_or_sync(FULL, n ? 1u << own : 0u);
  s.se += n && n < a.slot_n;
  // a wide slot's further 32 bytes are read here as well; where few lanes have more
  // than two of them, those lanes' slots, and rows longer than a slot, are put aside
  bool far = n >= (WIDE ? a.slot_n : CHUNK_IDS);
  if (WIDE) {
    const bool many = n >= 2 * CHUNK_IDS && !far;
    if (__popc(__ballot_sync(FULL, many)) < SLOT_LANES) far = far || many;
  }
  put_aside(a, s, far, own, u, n);
  if (far) n = 0;
  const uint32_t mx = __reduce_max_sync(FULL, n);
  uint32_t *row = reinterpret_cast<uint32_t *>(s_short + s.wb + own * a.Q);
  or_chunk(a, row, n, mx, first, second);
  // (put aside, two slots at a time by the whole warp, rows of 16 to 31 ids took twice
  // as long: 8,192 sources on the 10M-vertex power law, hop 4 30.5 -> 14.4 ms)
  if (WIDE)
    for (uint32_t i0 = CHUNK_IDS; i0 <= mx; i0 += CHUNK_IDS) {
      const bool on = n >= i0;
      uint4 x = make_uint4(0, 0, 0, 0), y = x;
      if (on) ld_slot(a.slot_in + (size_t)u * (a.slot_n / 8) + i0 / 8, x, y);
      const uint32_t z[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
#pragma unroll
      for (uint32_t i = 0; i < CHUNK_IDS; i++) {
        if (i0 + i > mx) break;
        const uint32_t id = i & 1 ? z[i >> 1] >> 16 : z[i >> 1] & 0xFFFFu;
        if (on && i0 + i <= n && may_grow(a, id)) or_id(row, id);
      }
    }
}

// The in-lists of the tile's targets, end to end (lane t: length deg of target t,
// which starts at entry `at` of adj; consecutive lists are consecutive there, a
// gap is a target that comes in pieces).  Rounds of G x 32 edges with their loads
// in flight at once; the warps of the SM cover the waits.
template <int MODE, int SLOTS, int T>
__device__ __forceinline__ void short_edges(const PullArgs &a, ShortEdges &s, const uint32_t *__restrict__ adj,
                                            int64_t at, uint32_t deg, bool gaps) {
  constexpr int G = SLOTS ? 2 : SH_GROUP;
  const uint32_t lane = threadIdx.x & 31, sq = a.slot_n / 8;
  // lane t: first edge of target t in the tile; lanes from T on: the number of edges
  uint32_t pre = deg;
#pragma unroll
  for (int o = 1; o < T; o <<= 1) {
    const uint32_t y = __shfl_up_sync(FULL, pre, o);
    if (lane >= o) pre += y;
  }
  const uint32_t total = __shfl_sync(FULL, pre, T - 1);
  pre = lane < T ? pre - deg : total;
  if (gaps) at -= pre;  // where target t's edges are, less their number in the tile
  else at = __shfl_sync(FULL, at, 0);
  for (uint32_t c = 0; c < total; c += 32 * G) {
    uint32_t u[G], own[G];
#pragma unroll
    for (int k = 0; k < G; k++) {
      const uint32_t e = c + k * 32 + lane;
      own[k] = 0;
#pragma unroll
      for (int step = T >> 1; step; step >>= 1)
        if (__shfl_sync(FULL, pre, own[k] + step) <= e) own[k] += step;
      const int64_t d = gaps ? __shfl_sync(FULL, at, own[k]) : at;
      u[k] = e < total ? __ldg(adj + d + e) : NONE;
    }
    if constexpr (!SLOTS) {
      Tiny w[G];
#pragma unroll
      for (int k = 0; k < G; k++) w[k] = u[k] != NONE ? ld_keep(a.tiny_in + u[k]) : 0u;
#pragma unroll
      for (int k = 0; k < G; k++) word_edges<MODE>(a, s, own[k], u[k], w[k]);
    } else {
      uint4 x[G], y[G];
#pragma unroll
      for (int k = 0; k < G; k++) {
        x[k] = y[k] = make_uint4(0, 0, 0, 0);
        if (u[k] != NONE) ld_slot(a.slot_in + (size_t)u[k] * sq, x[k], y[k]);
      }
#pragma unroll
      for (int k = 0; k < G; k++) slot_edges<MODE, SLOTS == 2>(a, s, own[k], u[k], x[k], y[k]);
    }
    drain<MODE>(a, s, c + 32 * G >= total);
  }
}

template <int MODE, int SLOTS, int T>
__device__ __forceinline__ void pull_short_run(const PullArgs &a, uint32_t wb) {
  const uint32_t lane = threadIdx.x & 31, Q = a.Q;
  uint4 *bm = s_short + wb;
  uint16_t *list = reinterpret_cast<uint16_t *>(bm + a.sh_list);
  uint8_t *before = reinterpret_cast<uint8_t *>(list);  // LAST: the cells' popcounts (at most 128)
  uint32_t *counts = reinterpret_cast<uint32_t *>(bm + a.sh_queue);
  const uint32_t ntasks = a.npieces + (a.V + T - 1) / T;
  // per thread: a warp's share of the rows, bits and edges of a layer that fits in
  // memory (V x W words) stays below 2^32; the product of degree and bits may not.  (All
  // in 64 bits spills: 1M- to 10M-vertex runs 2 to 4% slower.)
  unsigned long long po = 0;
  uint32_t nb = 0, nv = 0, nshort = 0, ntiny = 0, ro = 0, so = 0;
  ShortEdges s{wb, 0, 0, 0, 0, 0};
  auto fetch_task = [&]() { return lane == 0 ? atomicAdd(a.queue, 1u) : 0u; };
  uint32_t task = __shfl_sync(FULL, fetch_task(), 0);
  while (task < ntasks) {
    const uint32_t nexttask = fetch_task();  // in flight during this task
    s.whole = s.touched = 0;
    uint32_t v0;
    unsigned fm = 0;  // targets from v0 on to be done from their bitmaps
    uint32_t oldf = 0, total = 0;  // lane t: target t's flag (1: the buffer row holds an older layer's bits) and new bits
    if (task < a.npieces) {  // part of one long list
      const uint4 pc = __ldg(a.pieces + task);
      const uint32_t np = pc.y == NONE ? 1u : a.heavy_np[pc.y];
      for (uint32_t q = lane; q < Q; q += 32) bm[q] = make_uint4(0, 0, 0, 0);
      __syncwarp();
      const int64_t beg = a.in.off[pc.z][pc.x] + pc.w, end = a.in.off[pc.z][pc.x + 1];
      const uint32_t n = (uint32_t)min((int64_t)a.piece_edges, end - beg);
      short_edges<SH_GEN, SLOTS, 1>(a, s, a.in.adj[pc.z], beg, lane ? 0u : n, false);
      __syncwarp();  // every lane's ids are in the bitmap
      bool mine = true;
      if (np > 1) {
        uint4 *sum = a.heavy_rows + (size_t)pc.y * Q;
        for (uint32_t q = lane; q < Q; q += 32) add_union(sum + q, bm[q]);
        __threadfence();
        __syncwarp();
        uint32_t left = lane == 0 ? atomicSub(a.heavy_left + pc.y, 1u) : 0u;
        left = __shfl_sync(FULL, left, 0);
        mine = left == 1;
        if (mine) {  // the last piece: the whole union, and both left as they were found
          __threadfence();
          for (uint32_t q = lane; q < Q; q += 32) {
            bm[q] = __ldcg(sum + q);
            sum[q] = make_uint4(0, 0, 0, 0);
          }
          if (lane == 0) a.heavy_left[pc.y] = np;
        }
      }
      v0 = pc.x;
      fm = mine;
      if (fm) {
        oldf = a.flagN[v0];
        if (MODE != SH_LIST) total = new_bits<1>(a, wb, 1u, v0);
      }
    } else {
      v0 = (task - a.npieces) * T;
      const uint32_t v = v0 + lane;
      bool valid = lane < T && v < a.V, gaps = false;
      int64_t beg = 0;
      uint32_t deg = 0, rf = 0;
      if (valid) {
        beg = __ldg(a.in.off[0] + v);
        deg = (uint32_t)(__ldg(a.in.off[0] + v + 1) - beg);
        if (MODE != SH_GEN && a.shortest) rf = a.res_vis ? a.resflag[v] : 1u;
      }
      if (a.heavy_threshold) {
        uint64_t d = deg;
        if (valid && a.in.n > 1) d += (uint64_t)(__ldg(a.in.off[1] + v + 1) - __ldg(a.in.off[1] + v));
        const bool heavy = d > a.heavy_threshold;  // comes in pieces
        gaps = __any_sync(FULL, heavy);
        if (heavy) {
          valid = false;
          deg = rf = 0;
        }
      }
      if (MODE == SH_LIST && lane < T) counts[lane] = 0;
      {  // the bitmaps; resflag 0: the visited row is zero, without reading it
        const unsigned known = __ballot_sync(FULL, rf != 0);
        for (uint32_t q = lane; q < Q; q += 32) {
#pragma unroll
          for (int t0 = 0; t0 < T; t0 += T < 4 ? T : 4) {
            constexpr int B = T < 4 ? T : 4;  // rows with their loads in flight at once
            uint4 x[B];
#pragma unroll
            for (int t = 0; t < B; t++) {
              x[t] = make_uint4(0, 0, 0, 0);
              if (MODE != SH_GEN && (known >> (t0 + t) & 1u)) x[t] = a.vis[(size_t)(v0 + t0 + t) * Q + q];
            }
#pragma unroll
            for (int t = 0; t < B; t++) {
              bm[(t0 + t) * Q + q] = x[t];
              if (MODE == SH_LAST) before[(t0 + t) * Q + q] = (uint8_t)popc4(x[t]);
            }
          }
        }
      }
      __syncwarp();
#pragma unroll 1
      for (int l = 0; l < a.in.n; l++) {
        if (l) {
          if (lane < T && v < a.V) beg = __ldg(a.in.off[1] + v);
          if (valid) deg = (uint32_t)(__ldg(a.in.off[1] + v + 1) - beg);
        }
        short_edges<MODE, SLOTS, T>(a, s, l ? a.in.adj[1] : a.in.adj[0], beg, deg, gaps);
      }
      __syncwarp();
      if (valid) oldf = a.flagN[v];
      bool clean = valid && oldf == 1;                // ... and nothing will be written there
      if (MODE == SH_LAST) {
        const unsigned vm = __ballot_sync(FULL, valid);
        bool grew = false;
#pragma unroll
        for (int t = 0; t < T; t++) {
          if (!(vm >> t & 1u)) continue;
          bool any = false;
          for (uint32_t q0 = 0; q0 < Q; q0 += 32) {
            const uint32_t q = q0 + lane;
            uint4 x = make_uint4(0, 0, 0, 0);
            uint32_t more = 0;
            if (q < Q) {
              x = bm[t * Q + q];
              more = popc4(x) - before[t * Q + q];
            }
            nb += more;
            if (!__any_sync(FULL, more)) continue;
            if (q < Q) a.vis[(size_t)(v0 + t) * Q + q] = x;
            any = true;
          }
          if (lane == t) grew = any;
        }
        if (valid) {
          nv += grew;
          if (grew && a.res_vis) a.resflag[v] = 1;
          if (oldf) a.flagN[v] = 0;
        }
      } else {
        const uint32_t cnt = MODE == SH_LIST && lane < T ? counts[lane] : 0u;
        const bool from_row =
            valid && ((s.whole >> lane & 1u) || (MODE == SH_GEN ? (s.touched >> lane & 1u) : cnt >= a.slot_n));
        const bool listed = valid && !from_row;
        clean = clean && listed;
        fm = __ballot_sync(FULL, from_row);
        if (listed) {
          Tiny word = 0;
          if (MODE == SH_LIST && cnt) {
            uint16_t *li = list + lane * a.slot_n;
            li[0] = (uint16_t)cnt;
            word = tiny_word(cnt, cnt <= TINY_MAX ? li[1] | (cnt > 1 ? (uint32_t)li[2] << 15 : 0u) : 0u);
            if (a.res_vis) a.resflag[v] = 1;
            const uint32_t d = (uint32_t)out_degree(a.out, v);
            nb += cnt;
            nv++;
            nshort++;
            ntiny += cnt <= TINY_MAX;
            ro += d;
            so += d;
            po += (unsigned long long)d * cnt;
          }
          if (a.tiny_out) {
            a.tiny_out[v] = word;
            if (!cnt) a.slot_out[(size_t)v * a.slot_n] = 0;
          }
          const uint32_t nf = cnt ? 2u : 0u;
          if (nf != oldf) a.flagN[v] = nf;
        }
        if (MODE == SH_LIST) {
          const unsigned nm = __ballot_sync(FULL, listed && cnt);
          __syncwarp();
          const uint32_t sq = a.slot_n / 8, sh = 31 - __clz(sq);
          for (uint32_t i = lane; i < T * sq; i += 32)
            if (nm >> (i >> sh) & 1u)
              reinterpret_cast<uint4 *>(a.slot_out)[(size_t)v0 * sq + i] = reinterpret_cast<const uint4 *>(list)[i];
          if (a.shortest) {
#pragma unroll
            for (int t = 0; t < T; t++)
              if (nm >> t & 1u)
                for (uint32_t q = lane; q < Q; q += 32) a.vis[(size_t)(v0 + t) * Q + q] = bm[t * Q + q];
          }
        }
      }
      unsigned z = __ballot_sync(FULL, clean);
      while (z) {
        const uint32_t t = __ffs(z) - 1;
        z &= z - 1;
        for (uint32_t q = lane; q < Q; q += 32) a.N[(size_t)(v0 + t) * Q + q] = make_uint4(0, 0, 0, 0);
      }
      if (MODE == SH_GEN && fm) total = new_bits<T>(a, wb, fm, v0);
    }
    __syncwarp();
    while (fm) {
      const uint32_t t = __ffs(fm) - 1;
      fm &= fm - 1;
      if (MODE == SH_LIST) total = new_bits<1>(a, wb + t * Q, 1u, v0 + t);  // few: one at a time keeps the registers
      const uint32_t c = __shfl_sync(FULL, total, MODE == SH_LIST ? 0 : t);
      finish_row(a, wb, t, v0 + t, c, __shfl_sync(FULL, oldf, t));
      if (lane == 0 && c) {
        nb += c;
        nv++;
        if (a.tiny_out) {
          const uint32_t d = (uint32_t)out_degree(a.out, v0 + t);
          ro += d;
          po += (unsigned long long)d * c;
          if (c < a.slot_n) {
            nshort++;
            ntiny += c <= TINY_MAX;
            so += d;
          }
        }
      }
    }
    __syncwarp();
    task = __shfl_sync(FULL, nexttask, 0);
  }
  pull_counters(a, nb, nv, nshort + ((unsigned long long)ntiny << 32), s.se, ro, so, po);
}

// Layout of a warp's shared memory (uint4), and bytes of a block's.
inline void short_layout(PullArgs &a, uint32_t T) {
  a.sh_list = T * a.Q;
  a.sh_queue = a.sh_list + std::max(T * a.slot_n / 8, (T * a.Q + 15) / 16);  // lists, or a byte per cell
  a.sh_aside = a.sh_queue + (8 + SH_IDS) / 4;
  a.sh_warp = a.sh_aside + SH_ASIDE / 2;
}
constexpr uint32_t SHORT_MAX_Q = 256;  // cells of the widest rows (ids of 15 bits)
// Targets per tile: rows up to 1 KB four, wider ones two.
inline uint32_t short_tile(uint32_t Q) { return Q <= 64 ? 4 : 2; }
inline size_t short_smem(uint32_t Q, uint32_t slot_n) {
  PullArgs a;
  a.Q = Q;
  a.slot_n = slot_n;
  short_layout(a, short_tile(Q));
  return 16 * (2 * (size_t)Q + SH_WARPS * (size_t)a.sh_warp);
}

// The mode is the host's choice (short_kernel) except that a hop whose new rows
// will mostly be long finishes LIST as GEN; whether it reads words or slots is the
// device's: of the two kernels of a hop one returns at once (one kernel for both
// would need the registers of both).
template <int MODE, int SLOTS, int T>
__global__ void __launch_bounds__(SH_WARPS * 32, 4) k_pull_short(const __grid_constant__ PullArgs a) {
  vs::grid_wait();
  const HopCtr &hc = a.ctr->hop[a.h];
  if (hc.strategy != ST_PULL || !hc.short_pull || !a.tiny_in || (hc.short_slots != 0) != (SLOTS != 0) ||
      (MODE == SH_LIST && hc.short_long) || (MODE == SH_GEN && a.list_too && !hc.short_long))
    return;
  for (uint32_t q = threadIdx.x; q < a.Q; q += blockDim.x) {
    s_short[q] = make_uint4(0, 0, 0, 0);
    if (a.hmask) s_short[a.Q + q] = a.hmask[q];
  }
  __syncthreads();
  pull_short_run<MODE, SLOTS, T>(a, 2 * a.Q + (threadIdx.x >> 5) * a.sh_warp);
  __syncthreads();
  if (!a.last)
    for (uint32_t q = threadIdx.x; q < a.Q; q += blockDim.x) add_union(a.Uout + q, s_short[q]);
}

// Rows of layer h-1 left in their slots (flag 2), written out whole when hop
// h reads rows: a dense PULL or a PUSH (a short-mode PULL reads the slots).
// prev_virt: the PULL of hop h-1 was allowed to leave rows in their slots.
__device__ __forceinline__ void materialize(uint32_t *__restrict__ flagF, uint4 *__restrict__ F, uint32_t V, uint32_t Q,
                              const uint16_t *__restrict__ slots, uint32_t slot_n, const Ctr *ctr, int h,
                              int prev_virt) {
  const HopCtr &p = ctr->hop[h - 1], &c = ctr->hop[h];
  if (!prev_virt || p.strategy != ST_PULL || (p.short_rows & 0xFFFFFFFFull) == 0) return;
  if (c.strategy == 0 || (c.strategy == ST_PULL && c.short_pull)) return;
  const uint32_t lane = threadIdx.x & 31, warps = gridDim.x * (blockDim.x >> 5);
  for (uint32_t base = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * 32; base < V; base += warps * 32) {
    const uint32_t v = base + lane;
    const bool two = v < V && flagF[v] == 2;
    unsigned m = __ballot_sync(FULL, two);
    if (two) flagF[v] = 1;
    while (m) {
      // an id per lane into the row, which is zero, four rows' slots in flight at once
      uint32_t r[4], e[4];
#pragma unroll
      for (int k = 0; k < 4; k++) {
        r[k] = m ? base + __ffs(m) - 1 : NONE;
        m &= m - 1;
        e[k] = r[k] != NONE && lane < slot_n ? slots[(size_t)r[k] * slot_n + lane] : 0u;
      }
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const uint32_t cnt = __shfl_sync(FULL, e[k], 0);  // 0 past the last row
        uint32_t *row = reinterpret_cast<uint32_t *>(F + (size_t)r[k] * Q);
        if (lane && lane <= cnt) atomicOr(row + (e[k] >> 5), 1u << (e[k] & 31));
        if (lane + 32 <= cnt) {
          const uint32_t id = slots[(size_t)r[k] * slot_n + lane + 32];
          atomicOr(row + (id >> 5), 1u << (id & 31));
        }
      }
    }
  }
}

// Word and slot of row r held in one chunk (Q <= 32: lane q holds uint4 q).
__device__ __forceinline__ void short_from_chunk(uint4 x, uint32_t r, Tiny *tiny, uint16_t *slots,
                                                 uint32_t slot_n) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t n = popc4(x);
  uint32_t incl = n;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(FULL, incl, o);
    if (lane >= (uint32_t)o) incl += y;
  }
  const uint32_t total = __shfl_sync(FULL, incl, 31);
  uint32_t part = 0;  // ids 1 and 2 of the row, in tiny-word positions
  uint16_t *slot = slots + (size_t)r * slot_n;
  if (total < slot_n) {
    uint32_t at = 1 + incl - n;
    const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
    for (int wi = 0; wi < 4; wi++) {
      uint32_t bits = w[wi];
      while (bits) {
        const uint32_t t = __ffs(bits) - 1;
        bits &= bits - 1;
        const uint32_t id = lane * 128 + wi * 32 + t;
        if (at <= TINY_MAX) part |= id << (15 * (at - 1));
        slot[at] = (uint16_t)id;
        at++;
      }
    }
  }
  part = __reduce_or_sync(FULL, part);
  if (lane == 0) {
    tiny[r] = tiny_word(total, part);
    slot[0] = (uint16_t)(total < 0xFFFFu ? total : 0xFFFFu);
  }
}

// Hop h pulls in short mode over a layer that SPARSE (without overflow) or
// the seed wrote: that hop left exactly one (vertex, source) pair per bit, so
// the words and slots are built from the pair list instead of the rows.
__device__ __forceinline__ bool pairs_build(const Ctr *c, int h) {
  const HopCtr &cur = c->hop[h], &p = c->hop[h - 1];
  return cur.strategy == ST_PULL && cur.short_pull && (h == 1 || (p.strategy == ST_SPARSE && !p.overflow));
}

// Rows of a layer a SPARSE hop left in its pair list (Shortest: the hop
// dedups through the visited bits and writes no next-layer words), built
// before hop h reads them.  mode 0, right after hop h's decision: every pair
// when hop h reads whole rows (PUSH, dense or multi-slice PULL) or builds its
// short-row index from rows (the list overflowed); mode 1, after the index
// was built from the pairs: the pairs of rows too long for a slot, which a
// short-mode PULL gathers whole.  SPARSE reads only pairs.
__device__ __forceinline__ void pairs_rows(const uint2 *__restrict__ pairs, const uint32_t *__restrict__ cnt,
                             unsigned long long *__restrict__ N, uint32_t W, uint32_t slot_n, uint64_t cap,
                             const Ctr *ctr, int h, int mode) {
  if (ctr->hop[h - 1].strategy != ST_SPARSE) return;
  const int s = ctr->hop[h].strategy;
  const bool go = mode == 0 ? (s == ST_PUSH || (s == ST_PULL && !pairs_build(ctr, h))) : pairs_build(ctr, h);
  if (!go) return;
  const unsigned long long np_raw = ctr->hop[h - 1].pairs;
  const uint64_t np = np_raw < cap ? np_raw : cap;
  for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < np; k += (uint64_t)gridDim.x * blockDim.x) {
    const uint2 pr = pairs[k];
    if (mode == 1 && cnt[pr.x] < slot_n) continue;
    atomicOr(&N[(size_t)pr.x * W + (pr.y >> 6)], 1ull << (pr.y & 63));
  }
}

// every pair's source id into its vertex's slot (entries 1.., in any order)
__global__ void k_pairs_slots(const uint2 *__restrict__ pairs, uint32_t *__restrict__ cnt, uint16_t *__restrict__ slots,
                              uint32_t slot_n, uint64_t cap, const Ctr *ctr, int h) {
  vs::grid_wait();
  if (!pairs_build(ctr, h)) return;
  const unsigned long long np_raw = ctr->hop[h - 1].pairs;
  const uint64_t np = np_raw < cap ? np_raw : cap;
  for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < np; k += (uint64_t)gridDim.x * blockDim.x) {
    const uint2 pr = pairs[k];
    const uint32_t at = atomicAdd(&cnt[pr.x], 1u) + 1;
    if (at < slot_n) slots[(size_t)pr.x * slot_n + at] = (uint16_t)pr.y;
  }
}

// the tiny word of every vertex from its pair count (0 for an empty row)
__device__ __forceinline__ void pairs_words(const uint32_t *__restrict__ flagF, const uint32_t *__restrict__ cnt,
                              Tiny *__restrict__ tiny, uint16_t *__restrict__ slots, uint32_t slot_n, uint32_t V,
                              const Ctr *ctr, int h) {
  if (!pairs_build(ctr, h)) return;
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x) {
    const uint32_t c = flagF[v] ? cnt[v] : 0u;
    uint32_t part = 0;
    if (c && c <= TINY_MAX) {
      part = slots[(size_t)v * slot_n + 1];
      if (c > 1) part |= (uint32_t)slots[(size_t)v * slot_n + 2] << 15;
    }
    tiny[v] = tiny_word(c, part);
    if (c) slots[(size_t)v * slot_n] = (uint16_t)(c < 0xFFFFu ? c : 0xFFFFu);
  }
}

// Tiny words and slots of layer h-1 when hop h pulls in short mode and that
// layer was written by PUSH or by a SPARSE hop whose pair list overflowed: a warp per
// flagged row counts its bits and writes its word (and slot); every other
// vertex gets the count 0.
__device__ __forceinline__ void slot_build(const uint32_t *__restrict__ flagF, const uint4 *__restrict__ F, uint32_t V,
                             uint32_t Q, Tiny *__restrict__ tiny, uint16_t *__restrict__ slots, uint32_t slot_n,
                             const Ctr *ctr, int h) {
  if (ctr->hop[h].strategy != ST_PULL || !ctr->hop[h].short_pull || ctr->hop[h - 1].strategy == ST_PULL ||
      pairs_build(ctr, h))
    return;
  const int lane = threadIdx.x & 31;
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  for (uint32_t base = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * 32; base < V; base += warps * 32) {
    const uint32_t v = base + lane;
    const bool f = v < V && flagF[v];
    if (v < V && !f) {  // empty row
      tiny[v] = 0;
      slots[(size_t)v * slot_n] = 0;
    }
    unsigned m = __ballot_sync(FULL, f);
    if (Q <= 32) {  // one chunk per row: four rows' loads in flight at once
      while (m) {
        uint32_t rr[4] = {0, 0, 0, 0};
        int n = 0;
#pragma unroll
        for (int k = 0; k < 4; k++)
          if (m) {
            rr[k] = base + __ffs(m) - 1;
            m &= m - 1;
            n = k + 1;
          }
        uint4 x[4];
#pragma unroll
        for (int k = 0; k < 4; k++)
          x[k] = (k < n && (uint32_t)lane < Q) ? F[(size_t)rr[k] * Q + lane] : make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int k = 0; k < 4; k++)
          if (k < n) short_from_chunk(x[k], rr[k], tiny, slots, slot_n);
      }
      continue;
    }
    while (m) {
      const int b = __ffs(m) - 1;
      m &= m - 1;
      const uint32_t r = base + b;
      const uint4 *row = F + (size_t)r * Q;
      uint32_t c = 0;
      for (uint32_t q = lane; q < Q; q += 32) c += popc4(row[q]);
      const uint32_t total = warp_sum(c);
      uint32_t part = 0;  // ids 1 and 2 of the row, in tiny-word positions
      uint16_t *slot = slots + (size_t)r * slot_n;
      if (total < slot_n) {
        uint32_t pos = 1;
        for (uint32_t q0 = 0; q0 < Q; q0 += 32) {
          const uint32_t q = q0 + lane;
          const uint4 x = q < Q ? row[q] : make_uint4(0, 0, 0, 0);
          const uint32_t n = popc4(x);
          uint32_t incl = n;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(FULL, incl, o);
            if (lane >= o) incl += y;
          }
          uint32_t at = pos + incl - n;
          const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
          for (int wi = 0; wi < 4; wi++) {
            uint32_t bits = w[wi];
            while (bits) {
              const uint32_t t = __ffs(bits) - 1;
              bits &= bits - 1;
              const uint32_t id = q * 128 + wi * 32 + t;
              if (at <= TINY_MAX) part |= id << (15 * (at - 1));
              slot[at] = (uint16_t)id;
              at++;
            }
          }
          pos += __shfl_sync(FULL, incl, 31);
        }
      }
      part = __reduce_or_sync(FULL, part);
      if (lane == 0) {
        tiny[r] = tiny_word(total, part);
        slot[0] = (uint16_t)(total < 0xFFFFu ? total : 0xFFFFu);
      }
    }
  }
}

// Before hop h runs, in one launch: the rows of layer h-1 that its hop left in its
// pair list (deferred) or in their slots (virt), if hop h reads rows; the rows of
// layer h's buffer that an older layer left, if hop h needs them clean (SPARSE and
// PUSH write with atomics, a multi-slice PULL in parts; any PULL at hop 1 and later
// overwrites them itself); the pair counts of the short-row index; the row flags of
// layer h-1 as bits for a dense PULL that wants them.
struct PrepArgs {
  const uint2 *pairs;
  uint32_t *cnt;
  unsigned long long *F;
  uint32_t *flagF;
  uint4 *N;
  uint32_t *flagN;
  Tiny *tiny;
  uint16_t *slots;
  uint32_t *bits;
  uint32_t V, W, Q, slot_n;
  uint64_t cap;
  const Ctr *ctr;
  int h, deferred, virt, clear;
};

__global__ void __launch_bounds__(256) k_hop_prep(PrepArgs a) {
  vs::grid_wait();
  if (a.deferred) pairs_rows(a.pairs, a.cnt, a.F, a.W, a.slot_n, a.cap, a.ctr, a.h, 0);
  if (a.virt)
    materialize(a.flagF, reinterpret_cast<uint4 *>(a.F), a.V, a.Q, a.slots, a.slot_n, a.ctr, a.h, 1);
  const int s = a.ctr->hop[a.h].strategy;
  if (a.clear && (s == ST_SPARSE || s == ST_PUSH || (s == ST_PULL && a.ctr->multislice)))
    clear_flagged(a.N, a.flagN, a.V, a.Q);
  if (a.bits && a.ctr->hop[a.h].bits)
    for (uint32_t v0 = (blockIdx.x * blockDim.x + threadIdx.x) & ~31u; v0 < a.V; v0 += gridDim.x * blockDim.x) {
      const uint32_t v = v0 + (threadIdx.x & 31);
      const unsigned m = __ballot_sync(FULL, v < a.V && a.flagF[v]);
      if ((threadIdx.x & 31) == 0) a.bits[v0 >> 5] = m;
    }
  if (a.slots && pairs_build(a.ctr, a.h))
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < a.V; v += gridDim.x * blockDim.x) a.cnt[v] = 0;
}

// Short-row words of a layer SPARSE, PUSH or the seed wrote, from the pairs placed in
// the slots or from the rows, and the rows too long for a slot, which a short-mode
// PULL gathers whole.
__global__ void __launch_bounds__(256) k_short_index(PrepArgs a) {
  vs::grid_wait();
  pairs_words(a.flagF, a.cnt, a.tiny, a.slots, a.slot_n, a.V, a.ctr, a.h);
  if (a.deferred) pairs_rows(a.pairs, a.cnt, a.F, a.W, a.slot_n, a.cap, a.ctr, a.h, 1);
  slot_build(a.flagF, reinterpret_cast<const uint4 *>(a.F), a.V, a.Q, a.tiny, a.slots, a.slot_n, a.ctr, a.h);
}

// ---------------------------------------------------------------------------
// PUSH.  Active rows of layer h-1 (flag set) are compacted into a list; a warp
// per active vertex ORs its row into each out-neighbour's next-layer row with
// 64-bit atomics and records first touches; a second pass over the touched
// list applies the visited AND-NOT and the accumulator (Shortest/Any rules).
__global__ void k_push_compact(const uint32_t *__restrict__ flagF, uint32_t V, uint32_t *list,
                               Ctr *ctr, int h) {
  vs::grid_wait();
  if (ctr->hop[h].strategy != ST_PUSH) return;
  const int lane = threadIdx.x & 31;
  for (uint32_t v0 = (blockIdx.x * blockDim.x + threadIdx.x) & ~31u; v0 < V;
       v0 += gridDim.x * blockDim.x) {
    const uint32_t v = v0 + lane;
    const bool f = v < V && flagF[v];
    const unsigned m = __ballot_sync(FULL, f);
    if (!m) continue;
    unsigned base = 0;
    if (lane == 0) base = atomicAdd(&ctr->push_active, (unsigned)__popc(m));
    base = __shfl_sync(FULL, base, 0);
    if (f) list[base + __popc(m & lanemask_lt())] = v;
  }
}

__global__ void __launch_bounds__(256) k_push(PushArgs a) {
  vs::grid_wait();
  Ctr *c = a.ctr;
  if (c->hop[a.h].strategy != ST_PUSH) return;
  const uint32_t n = c->push_active;
  const int lane = threadIdx.x & 31;
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  for (uint32_t t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); t < n; t += warps) {
    const uint32_t u = a.active[t];
    const unsigned long long *row = a.F + (size_t)u * a.W;
    _Pragma("unroll") for (int l = 0; l < 2; l++) if (l < a.out.n) {
      const int64_t beg = a.out.off[l][u], end = a.out.off[l][u + 1];
      for (int64_t j = beg; j < end; j++) {
        const uint32_t v = __ldg(a.out.adj[l] + j);
        unsigned long long *dst = a.N + (size_t)v * a.W;
        for (uint32_t w = lane; w < a.W; w += 32) {
          const unsigned long long x = row[w];
          if (x) atomicOr(dst + w, x);
        }
        if (lane == 0 && atomicOr(&a.flagN[v], 1u) == 0) {
          unsigned s = atomicAdd(&c->push_touched, 1u);
          a.touched[s] = v;
        }
      }
    }
  }
}

__global__ void __launch_bounds__(256) k_push_epilogue(PushArgs a) {
  vs::grid_wait();
  Ctr *c = a.ctr;
  if (c->hop[a.h].strategy != ST_PUSH) return;
  const uint32_t n = c->push_touched;
  const int lane = threadIdx.x & 31;
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  unsigned long long nb = 0, nv = 0;
  for (uint32_t t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); t < n; t += warps) {
    const uint32_t v = a.touched[t];
    bool any = false;
    for (uint32_t w = lane; w < a.W; w += 32) {
      const size_t idx = (size_t)v * a.W + w;
      unsigned long long x = a.N[idx];
      const unsigned long long x0 = x;
      if (a.hmask) x &= a.hmask[w];
      if (a.shortest && x) {
        const unsigned long long vv = a.vis[idx];
        x &= ~vv;
        if (x) a.vis[idx] = vv | x;
      }
      if (x != x0) a.N[idx] = x;
      if (x) {
        any = true;
        nb += __popcll(x);
        if (a.acc_on) a.acc[idx] |= x;
      }
    }
    const bool rownz = __any_sync(FULL, any);
    if (lane == 0) {
      if (!rownz)
        a.flagN[v] = 0;  // row is all zero again
      else
        nv++;
      if (rownz && (a.res_vis || a.acc_on)) a.resflag[v] = 1;
    }
  }
  block_add(nb, &c->hop[a.h].new_bits);
  block_add(nv, &c->hop[a.h].active_vertices);
}

__global__ void k_push_reset(Ctr *c) {
  vs::grid_wait();
  c->push_active = 0;
  c->push_touched = 0;
}

// FindShortest target check of hop h (vexpand.cpp:237-271).
__global__ void k_find_check(const uint64_t *__restrict__ N, const uint32_t *__restrict__ tgt,
                             int32_t *__restrict__ dist, uint32_t S, uint32_t W, uint32_t V,
                             Ctr *ctr, int h) {
  vs::grid_wait();
  if (ctr->hop[h].strategy == 0) return;
  unsigned long long f = 0;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < S; i += gridDim.x * blockDim.x) {
    if (tgt[i] < V && dist[i] == -1 && ((N[(size_t)tgt[i] * W + (i >> 6)] >> (i & 63)) & 1ull)) {
      dist[i] = h;
      f++;
    }
  }
  block_add(f, &ctr->found);
}

// Shortest with k_min == 1: the result is visited minus layer 0, i.e. the
// source bits (i, s_i) cleared (a source is never re-reached once visited).
__global__ void k_clear_diag(uint64_t *__restrict__ vis, const uint32_t *__restrict__ src,
                             uint32_t S, uint32_t W, uint32_t V) {
  vs::grid_wait();
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < S; i += gridDim.x * blockDim.x)
    if (src[i] < V) atomicAnd((unsigned long long *)&vis[(size_t)src[i] * W + (i >> 6)], ~(1ull << (i & 63)));
}

// Targets of a direction set whose in-degree is above the threshold: their list
// (n[0]), the pieces the dense PULL cuts them into (n[1]) and how many have more
// than one (n[2]).
__device__ __forceinline__ uint32_t pieces_of(const Lists &in, uint32_t v, int l, uint32_t piece) {
  return l < in.n ? (uint32_t)((in.off[l][v + 1] - in.off[l][v] + piece - 1) / piece) : 0u;
}

__global__ void k_hubs(Lists in, uint32_t V, uint32_t thr, uint32_t piece, uint32_t *list, unsigned *n) {
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x) {
    int64_t d = 0;
    _Pragma("unroll") for (int l = 0; l < 2; l++) if (l < in.n) d += in.off[l][v + 1] - in.off[l][v];
    if (d <= (int64_t)thr) continue;
    list[atomicAdd(n, 1u)] = v;
    const uint32_t np = pieces_of(in, v, 0, piece) + pieces_of(in, v, 1, piece);
    atomicAdd(n + 1, np);
    if (np > 1) atomicAdd(n + 2, 1u);
  }
}

// n[0] pieces and n[1] targets of several pieces written so far
__global__ void k_hub_pieces(Lists in, const uint32_t *__restrict__ heavy, uint32_t nheavy, uint32_t piece,
                             uint4 *__restrict__ pieces, unsigned *n, uint32_t *__restrict__ np_of,
                             uint32_t *__restrict__ left, uint32_t nslices) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nheavy; i += gridDim.x * blockDim.x) {
    const uint32_t v = heavy[i];
    const uint32_t np[2] = {pieces_of(in, v, 0, piece), pieces_of(in, v, 1, piece)};
    uint32_t row = NONE;
    if (np[0] + np[1] > 1) {
      row = atomicAdd(n + 1, 1u);
      np_of[row] = np[0] + np[1];
      for (uint32_t y = 0; y < nslices; y++) left[(size_t)row * nslices + y] = np[0] + np[1];
    }
    uint32_t at = atomicAdd(n, np[0] + np[1]);
    for (uint32_t l = 0; l < 2; l++)
      for (uint32_t k = 0; k < np[l]; k++) pieces[at++] = make_uint4(v, row, l, k * piece);
  }
}

// ---------------------------------------------------------------------------
// Host side.

Lists pull_lists(const vs_graph *g, int dir) {
  Lists L;
  L.n = 0;
  const bool fwd = !g->directed || dir == VS_DIR_FORWARD || dir == VS_DIR_BOTH;
  const bool bwd = g->directed && (dir == VS_DIR_BACKWARD || dir == VS_DIR_BOTH);
  if (fwd) {  // in-lists of the target: reverse CSR
    L.off[L.n] = g->rev_off;
    L.adj[L.n] = g->rev_src;
    L.n++;
  }
  if (bwd) {
    L.off[L.n] = g->fwd_off;
    L.adj[L.n] = g->fwd_dst;
    L.n++;
  }
  return L;
}

Lists push_lists(const vs_graph *g, int dir) {
  Lists L;
  L.n = 0;
  const bool fwd = !g->directed || dir == VS_DIR_FORWARD || dir == VS_DIR_BOTH;
  const bool bwd = g->directed && (dir == VS_DIR_BACKWARD || dir == VS_DIR_BOTH);
  if (fwd) {
    L.off[L.n] = g->fwd_off;
    L.adj[L.n] = g->fwd_dst;
    L.n++;
  }
  if (bwd) {
    L.off[L.n] = g->rev_off;
    L.adj[L.n] = g->rev_src;
    L.n++;
  }
  return L;
}

using PullFn = void (*)(PullArgs);

// Short-mode kernels of a row width: words and slots by mode (a slot hop has no LIST).
// Slots of 16 entries have kernels of their own: the second piece of a wider one,
// never there, cost 4% of a 14 ms run in registers and code.
struct ShortVariant {
  uint32_t T;
  PullFn words[3], slots[3];
};
#define VS_SHORT(T, K) \
  {T, {k_pull_short<SH_LIST, 0, T>, k_pull_short<SH_LAST, 0, T>, k_pull_short<SH_GEN, 0, T>}, \
   {nullptr, k_pull_short<SH_LAST, K, T>, k_pull_short<SH_GEN, K, T>}}
const ShortVariant kShort[3] = {VS_SHORT(4, 1), VS_SHORT(4, 2), VS_SHORT(2, 2)};
#undef VS_SHORT
const ShortVariant &pick_short(uint32_t Q, uint32_t slot_n) {
  return kShort[short_tile(Q) == 2 ? 2 : slot_n > CHUNK_IDS ? 1 : 0];
}

struct PullVariant {
  int L, UPL;
  PullFn pull, bits;
};

#define VS_VARIANT(L) {L, 1, k_pull<L, 1, false>, k_pull<L, 1, true>}
#define VS_WIDE(U) {32, U, k_pull<32, U, false>, nullptr}  // L = 32: 1% slower with bits on power laws
const PullVariant kVariants[] = {VS_VARIANT(1),  VS_VARIANT(2), VS_VARIANT(4), VS_VARIANT(8), VS_VARIANT(16),
                                 VS_WIDE(1),     VS_WIDE(2),    VS_WIDE(4),    VS_WIDE(8)};
#undef VS_VARIANT
#undef VS_WIDE

const PullVariant &pick_variant(uint32_t qslice) {
  for (const auto &v : kVariants)
    if ((uint32_t)(v.L * v.UPL) >= qslice) return v;
  return kVariants[sizeof(kVariants) / sizeof(kVariants[0]) - 1];
}

}  // namespace ex
}  // namespace vs

using namespace vs;
using namespace vs::ex;

struct vs_expand_plan {
  vs_graph *g = nullptr;
  vs_expand_params p{};
  uint32_t S = 0, W = 0, Q = 0, qslice = 0, nslices = 1;
  uint64_t *buf[2] = {nullptr, nullptr};
  uint32_t *flag[2] = {nullptr, nullptr};
  uint32_t *bits = nullptr;  // row flags of the layer a dense PULL reads
  uint64_t *vis = nullptr, *acc = nullptr;
  uint2 *pairs[2] = {nullptr, nullptr};
  unsigned long long *pdeg[2] = {nullptr, nullptr}, *doff = nullptr, *bsum = nullptr;
  uint64_t pair_cap = 0;
  uint32_t *push_list = nullptr, *touched = nullptr;
  uint32_t *resflag = nullptr;  // per vertex: result column may be non-zero
  uint32_t *d_src = nullptr, *d_tgt = nullptr;
  int32_t *d_dist = nullptr;
  Ctr *ctr = nullptr;
  // PULL: targets above heavy_threshold are cut into pieces
  uint32_t heavy_threshold = 0, nheavy = 0, npieces = 0, tile = 32;
  uint4 *pieces = nullptr, *heavy_rows = nullptr;
  uint32_t *heavy_np = nullptr, *heavy_left = nullptr;
  uint4 *un = nullptr;         // (k_max + 1) x Q uint4: union of the rows of every layer a PULL hop wrote
  uint32_t *queue = nullptr;   // (k_max + 1) x nslices task counters of the PULL hops
  size_t ctr_bytes = 0;        // ctr, un and queue are one allocation, zeroed at every run start
  bool use_vis = false, use_acc = false, clear_diag = false;
  bool collect_stats = false;
  int grid_bits = 0, grid_pull = 0, grid_sparse = 0, grid_v = 0, grid_push = 0, grid_short = 0;
  vs_bitmat result{};
  bool has_result = false;
  // tuning knobs of the fixed planner
  double sparse_frac = 0.02, push_frac = 0.0;
  const void *picker = nullptr;
  bool log_features = false;
  uint64_t *hmask = nullptr;  // (k_max + 1) x W words: rows allowed to grow at hop h
  uint32_t *rowk = nullptr;   // [0] largest row limit, [1] a limit exceeded k_max (device-set limits)
  uint64_t *layer_out[VS_MAX_HOPS + 1] = {};  // with_distance: layer h is copied here (zeroed, V x W words)
  // short-row index of the two frontier buffers' layers; none when S > 32768 or multi-slice
  Tiny *tiny[2] = {nullptr, nullptr};      // short-row words
  uint16_t *slot[2] = {nullptr, nullptr};  // ... and their slots
  uint32_t slot_n = 16;                    // uint16 entries per slot
  double short_min = 0.0;                  // share of short rows for a short-mode PULL (0: off)
  bool use_hmask = false;
  int hop_forced[VS_MAX_HOPS + 1] = {};
  bool timing = false;
  uint32_t timed_hops = 0;
  cudaStream_t last_stream = 0;  // frees are ordered after the last run on it
  cudaEvent_t ev[3 * (VS_MAX_HOPS + 1)] = {};
  // one-shot cache: the caller's parameters, the graph's serial, the plan's
  // device bytes and the event its last user's stream recorded
  vs_expand_params key{};
  uint64_t graph_serial = 0, bytes = 0;
  cudaEvent_t cache_ev = nullptr;
};

namespace vs {
namespace ex {

// Any with k_min == k_max returns layer k_max itself: no accumulator (the last
// frontier buffer is the result).  Any over a range, and Shortest with
// k_min >= 2, union layers k_min..k_max into an accumulator.
inline bool needs_acc(const vs_expand_params &p) {
  return (p.path_type == VS_PATH_ANY && p.k_min != p.k_max) ||
         (p.path_type == VS_PATH_SHORTEST && p.k_min >= 2);
}

// uint16 entries of a short-row slot for rows of W words: a sixteenth of
// the row's bytes at 64 and 128 words, 128 bytes beyond.
inline uint32_t slot_entries(uint32_t W) { return W <= 64 ? 16 : W <= 128 ? 32 : 64; }

// Short-row words and slots (15-bit ids: S <= 32768) need rows in one slice.
// Short mode is not worth them on a graph whose whole V x W matrix fits in half
// of L2, nor for rows below 32 words: a dense hop of 16-word rows took 0.25 ms on
// the 1M-vertex power law where a short one took 0.38 (unless forced: share > 1).
inline bool short_slots_ok(uint32_t S, uint32_t nslices, double share, uint64_t V, uint32_t W) {
  return share >= 0 && S <= 128 * SHORT_MAX_Q && nslices == 1 && (share > 1.0 || (W >= 32 && V * 8ull * W > l2_bytes() / 2));
}

// Whether a plan's dense PULL hops may read row flags as bits.  Whole runs against flags
// in global memory, power laws and R-MAT graphs of 16K to 1.2M vertices: rows of 3 to 16
// uint4 gain 3 to 16% from 128K vertices on and lose up to 5% at 16K to 64K (the block's
// prologue and one launch a hop); rows of one or two gain 2 to 23% at 18M list entries
// and more and lose 1 to 5% at 4M to 8M; rows of 32 lanes lose 1% on power laws.
inline bool bits_ok(uint32_t V, uint32_t qslice, bool slots, uint64_t list_edges) {
  const PullVariant &v = pick_variant(qslice);
  if (!v.bits || V > BITS_MAX_V || (slots && v.L < 16)) return false;  // (no room to write slots in narrow rows)
  return v.L <= 2 ? list_edges >= BITS_MIN_EDGES : V >= BITS_MIN_V;
}

int plan_free(vs_expand_plan *pl) {
  if (!pl) return VS_OK;
  const cudaStream_t st = pl->last_stream;
  void *ptrs[] = {pl->tiny[0], pl->tiny[1], pl->slot[0], pl->slot[1], pl->resflag, pl->pdeg[0], pl->pdeg[1], pl->doff,
                  pl->bsum, pl->hmask, pl->rowk, pl->buf[0], pl->buf[1], pl->flag[0], pl->flag[1], pl->vis, pl->acc,
                  pl->pairs[0], pl->pairs[1], pl->push_list, pl->touched, pl->d_src,
                  pl->d_tgt, pl->d_dist, pl->ctr, pl->pieces, pl->bits};
  for (void *p : ptrs)  // stream-ordered after the plan's last run
    if (p) dfree(p, st);
  for (cudaEvent_t e : pl->ev)
    if (e) cudaEventDestroy(e);
  if (pl->cache_ev) cudaEventDestroy(pl->cache_ev);
  delete pl;
  return VS_OK;
}

// The one-shot vs_expand keeps its plans: a call takes an idle plan built for
// the same graph, source count and parameters (or builds one), runs it and
// hands out the result as a view whose release returns the plan.  Reuse skips
// the allocations, the full-matrix clears of a new plan and its hub list; a
// run clears only what the previous run wrote.  At most kCacheIdle idle plans
// are kept, holding at most a quarter of the device's memory (48 GB at
// least); vs_release_cached frees them all.
constexpr size_t kCacheIdle = 8;

uint64_t cache_bytes_cap() {
  static uint64_t cap = 0;
  if (cap == 0) {
    size_t free_b = 0, total_b = 0;
    cap = 48ull << 30;
    if (cudaMemGetInfo(&free_b, &total_b) == cudaSuccess) cap = std::max<uint64_t>(cap, total_b / 4);
  }
  return cap;
}

struct PlanCache {
  std::mutex mu;
  std::vector<vs_expand_plan *> idle;  // oldest first
  std::vector<uint64_t> dead;          // serials of freed graphs (plans lent out then are freed on return)
};
PlanCache &plan_cache() {
  static PlanCache c;
  return c;
}

bool same_params(const vs_expand_params &a, const vs_expand_params &b) {
  return a.k_min == b.k_min && a.k_max == b.k_max && a.path_type == b.path_type && a.direction == b.direction &&
         a.strategy == b.strategy && a.use_picker == b.use_picker && a.hub_threshold == b.hub_threshold &&
         a.slice_words == b.slice_words && a.pair_capacity == b.pair_capacity &&  // (pull_kernel has no effect)
         a.sparse_frac == b.sparse_frac && a.short_share == b.short_share;
}

vs_expand_plan *plan_cache_take(const vs_graph *g, uint32_t S, const vs_expand_params &p) {
  PlanCache &c = plan_cache();
  std::lock_guard<std::mutex> lk(c.mu);
  for (size_t i = c.idle.size(); i-- > 0;) {
    vs_expand_plan *pl = c.idle[i];
    if (pl->graph_serial == g->serial && pl->S == S && same_params(pl->key, p)) {
      c.idle.erase(c.idle.begin() + (long)i);
      return pl;
    }
  }
  return nullptr;
}

void plan_cache_trim(PlanCache &c, std::vector<vs_expand_plan *> &drop) {
  uint64_t bytes = 0;
  for (vs_expand_plan *pl : c.idle) bytes += pl->bytes;
  const uint64_t cap = cache_bytes_cap();
  while (!c.idle.empty() && (c.idle.size() > kCacheIdle || bytes > cap)) {
    bytes -= c.idle.front()->bytes;
    drop.push_back(c.idle.front());
    c.idle.erase(c.idle.begin());
  }
}

}  // namespace ex

uint64_t next_graph_serial() {
  static std::atomic<uint64_t> n{1};
  return n++;
}

void plan_cache_return(vs_expand_plan *pl, cudaStream_t st) {
  using namespace ex;
  if (!pl->cache_ev) cudaEventCreateWithFlags(&pl->cache_ev, cudaEventDisableTiming);
  if (pl->cache_ev) cudaEventRecord(pl->cache_ev, st);  // the next user's stream waits for this one
  pl->last_stream = st;
  std::vector<vs_expand_plan *> drop;
  {
    PlanCache &c = plan_cache();
    std::lock_guard<std::mutex> lk(c.mu);
    if (std::find(c.dead.begin(), c.dead.end(), pl->graph_serial) != c.dead.end() || !pl->cache_ev) {
      drop.push_back(pl);
    } else {
      c.idle.push_back(pl);
      plan_cache_trim(c, drop);
    }
  }
  for (vs_expand_plan *d : drop) plan_free(d);
}

void plan_cache_drop_graph(uint64_t serial) {
  using namespace ex;
  std::vector<vs_expand_plan *> drop;
  {
    PlanCache &c = plan_cache();
    std::lock_guard<std::mutex> lk(c.mu);
    c.dead.push_back(serial);
    for (size_t i = 0; i < c.idle.size();) {
      if (c.idle[i]->graph_serial == serial) {
        drop.push_back(c.idle[i]);
        c.idle.erase(c.idle.begin() + (long)i);
      } else {
        i++;
      }
    }
  }
  for (vs_expand_plan *d : drop) plan_free(d);
}

namespace ex {

template <typename K> int occupancy_grid(K kernel, int threads, size_t smem, int cap_per_sm) {
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem);
  if (per_sm <= 0) per_sm = 1;
  if (cap_per_sm > 0 && per_sm > cap_per_sm) per_sm = cap_per_sm;
  return per_sm * sm_count();
}

}  // namespace ex
}  // namespace vs

extern "C" {

int vs_expand_plan_create(vs_graph *g, uint32_t S, const vs_expand_params *p,
                          vs_expand_plan **out) {
  if (!g || !p || !out) return fail(VS_ERR_ARG, "vs_expand_plan_create: null argument");
  if (p->k_min > p->k_max) return fail(VS_ERR_ARG, "k_min %u > k_max %u", p->k_min, p->k_max);
  if (p->k_max > VS_MAX_HOPS) return fail(VS_ERR_ARG, "k_max %u exceeds %d", p->k_max, VS_MAX_HOPS);
  if (p->path_type < VS_PATH_ANY || p->path_type > VS_PATH_FIND_SHORTEST)
    return fail(VS_ERR_ARG, "unknown path type %d", p->path_type);
  if (p->direction < VS_DIR_FORWARD || p->direction > VS_DIR_BOTH)
    return fail(VS_ERR_ARG, "unknown direction %d", p->direction);
  if (p->strategy < VS_STRAT_AUTO || p->strategy > VS_STRAT_SPARSE)
    return fail(VS_ERR_ARG, "unknown strategy %d", p->strategy);
  if (p->pull_kernel < 0 || p->pull_kernel > 7) return fail(VS_ERR_ARG, "pull kernel variant must be 0..7");
  if (p->sparse_frac < 0) return fail(VS_ERR_ARG, "sparse_frac must be >= 0");
  if (S == 0) return fail(VS_ERR_ARG, "no start vertex for VExpand");
  if (S >= 0x80000000u) return fail(VS_ERR_ARG, "VExpand takes fewer than 2^31 start vertices");
  cudaStream_t st = 0;
  vs_expand_plan *pl = new vs_expand_plan();
  pl->g = g;
  pl->p = *p;
  pl->S = S;
  pl->W = words_per_col(S);
  pl->Q = pl->W / 2;
  uint32_t qs = p->slice_words ? (p->slice_words + 1) / 2 : pl->Q;
  qs = std::min(qs, (uint32_t)256);
  if (qs == 0) qs = 1;
  pl->qslice = qs;
  pl->nslices = (pl->Q + qs - 1) / qs;
  const bool shortest = p->path_type != VS_PATH_ANY;
  pl->use_vis = shortest;
  pl->use_acc = needs_acc(*p);
  pl->clear_diag = p->path_type == VS_PATH_SHORTEST && p->k_min == 1;
  const uint32_t V = g->V;
  const size_t rowwords = (size_t)V * pl->W;
  pl->pair_cap = p->pair_capacity ? p->pair_capacity
                                  : std::max<uint64_t>(1u << 20, std::min<uint64_t>((uint64_t)S * V / 8, 1ull << 25));
  pl->pair_cap = std::max<uint64_t>(pl->pair_cap, S);
  int rc = VS_OK;
#define PL_ALLOC(ptr, n)                                          \
  if ((rc = dalloc_n(&(ptr), (n), st)) != VS_OK) {                \
    plan_free(pl);                                                \
    return rc;                                                    \
  }
  PL_ALLOC(pl->buf[0], rowwords);
  PL_ALLOC(pl->buf[1], rowwords);
  PL_ALLOC(pl->flag[0], V);
  PL_ALLOC(pl->flag[1], V);
  if (pl->use_vis) PL_ALLOC(pl->vis, rowwords);
  if (pl->use_acc) PL_ALLOC(pl->acc, rowwords);
  PL_ALLOC(pl->pairs[0], pl->pair_cap);
  PL_ALLOC(pl->pairs[1], pl->pair_cap);
  PL_ALLOC(pl->pdeg[0], pl->pair_cap);
  PL_ALLOC(pl->pdeg[1], pl->pair_cap);
  PL_ALLOC(pl->doff, pl->pair_cap + 1);
  PL_ALLOC(pl->bsum, (pl->pair_cap + 1023) / 1024 + 1);
  PL_ALLOC(pl->push_list, V);
  PL_ALLOC(pl->resflag, V);
  PL_ALLOC(pl->touched, V);
  PL_ALLOC(pl->d_src, S);
  if (p->path_type == VS_PATH_FIND_SHORTEST) {
    PL_ALLOC(pl->d_tgt, S);
    PL_ALLOC(pl->d_dist, S);
  }
  {  // counters, layer unions and task queues in one block, which a run's first kernel clears
    const size_t c = (sizeof(Ctr) + 15) / 16 * 16, u = (size_t)(p->k_max + 1) * pl->Q * 16;
    pl->ctr_bytes = (c + u + (size_t)(p->k_max + 1) * pl->nslices * 4 + 15) / 16 * 16;
    char *base = nullptr;
    PL_ALLOC(base, pl->ctr_bytes);
    pl->ctr = reinterpret_cast<Ctr *>(base);
    pl->un = reinterpret_cast<uint4 *>(base + c);
    pl->queue = reinterpret_cast<uint32_t *>(base + c + u);
  }
  PL_ALLOC(pl->hmask, (size_t)(p->k_max + 1) * pl->W);
  PL_ALLOC(pl->rowk, 2);
  pl->short_min = p->short_share == 0 ? 0.1 : p->short_share;
  if (short_slots_ok(S, pl->nslices, p->short_share, V, pl->W)) {
    PL_ALLOC(pl->tiny[0], V);
    PL_ALLOC(pl->tiny[1], V);
    pl->slot_n = slot_entries(pl->W);
    PL_ALLOC(pl->slot[0], (size_t)V * pl->slot_n);
    PL_ALLOC(pl->slot[1], (size_t)V * pl->slot_n);
  } else {
    pl->short_min = 0;
  }
  if (bits_ok(V, pl->qslice, pl->slot[0] != nullptr, (p->direction == VS_DIR_BOTH && g->directed ? 2 : 1) * g->E)) PL_ALLOC(pl->bits, bits_smem(V) / 4);
#undef PL_ALLOC
  cudaError_t e = cudaSuccess;
  // every row starts zero; later runs clear only the rows their flags mark
  if ((e = cudaMemsetAsync(pl->buf[0], 0, rowwords * 8, st)) != cudaSuccess ||
      (e = cudaMemsetAsync(pl->buf[1], 0, rowwords * 8, st)) != cudaSuccess ||
      (e = cudaMemsetAsync(pl->flag[0], 0, 4ull * V, st)) != cudaSuccess ||
      (e = cudaMemsetAsync(pl->flag[1], 0, 4ull * V, st)) != cudaSuccess ||
      (e = cudaMemsetAsync(pl->resflag, 0, 4ull * V, st)) != cudaSuccess ||
      (pl->vis && (e = cudaMemsetAsync(pl->vis, 0, rowwords * 8, st)) != cudaSuccess) ||
      (pl->acc && (e = cudaMemsetAsync(pl->acc, 0, rowwords * 8, st)) != cudaSuccess)) {
    plan_free(pl);
    return cuda_fail(e, "cudaMemsetAsync", __FILE__, __LINE__);
  }
  // heavy targets of the pull direction set and their pieces
  const PullVariant &var = pick_variant(pl->qslice);
  pl->heavy_threshold = p->hub_threshold ? std::min(p->hub_threshold, HEAVY_MAX) : heavy_default(var.L);
  {
    Lists in = pull_lists(g, p->direction);
    unsigned *dn = nullptr;  // counters, then the heavy targets
    if ((rc = dalloc_n(&dn, 8 + (size_t)V, st)) != VS_OK) {
      plan_free(pl);
      return rc;
    }
    uint32_t *heavy = dn + 8;
    cudaMemsetAsync(dn, 0, 8 * sizeof(unsigned), st);
    const uint32_t pe = piece_edges(var.L);
    { k_hubs<<<sm_count() * 4, 256, 0, st>>>(in, V, pl->heavy_threshold, pe, heavy, dn); vs::note_launch(); }
    unsigned hn[3] = {0, 0, 0};
    cudaMemcpyAsync(hn, dn, sizeof(hn), cudaMemcpyDeviceToHost, st);
    e = cudaStreamSynchronize(st);
    pl->nheavy = hn[0];
    pl->npieces = hn[1];
    const size_t nmulti = hn[2];
    if (e == cudaSuccess && pl->nheavy) {  // one allocation: pieces, unions, counts
      const size_t rows = nmulti * pl->Q, first = ((size_t)pl->npieces + 15) / 16 * 16;  // rows of whole lines
      if ((rc = dalloc_n(&pl->pieces, first + rows + (nmulti * (1 + pl->nslices) + 3) / 4, st)) != VS_OK) {
        dfree(dn, st);
        plan_free(pl);
        return rc;
      }
      pl->heavy_rows = pl->pieces + first;
      pl->heavy_np = reinterpret_cast<uint32_t *>(pl->heavy_rows + rows);
      pl->heavy_left = pl->heavy_np + nmulti;
      e = cudaMemsetAsync(pl->heavy_rows, 0, rows * 16, st);
      // (a first run on another stream waits for this one)
      { k_hub_pieces<<<sm_count() * 4, 256, 0, st>>>(in, heavy, pl->nheavy, pe, pl->pieces, dn + 3, pl->heavy_np,
                                                     pl->heavy_left, pl->nslices); vs::note_launch(); }
      if (e == cudaSuccess) e = cudaGetLastError();
    }
    dfree(dn, st);
    if (e != cudaSuccess) {
      plan_free(pl);
      return cuda_fail(e, "hub list", __FILE__, __LINE__);
    }
  }
  if (p->sparse_frac > 0) pl->sparse_frac = p->sparse_frac;
  // a task is `tile` consecutive targets: a round of the warp's groups on small
  // graphs (more tasks than warps), up to 16 targets on large ones
  const uint32_t G = 32 / var.L;
  const int occ = occupancy_grid(var.pull, 256, 0, 8);
  pl->tile = G;
  while (pl->tile < 16 && (uint64_t)V / pl->tile > 64ull * occ) pl->tile *= 2;
  if (pl->bits) {
    cudaFuncSetAttribute(var.bits, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bits_smem(BITS_MAX_V));
    pl->grid_bits = occupancy_grid(var.bits, 1024, bits_smem(V), 1);
  }
  const uint64_t tasks = pl->npieces + ((uint64_t)V + pl->tile - 1) / pl->tile;
  pl->grid_pull = (int)std::max<uint64_t>(1, std::min<uint64_t>(occ, (tasks + 7) / 8));
  if (pl->slot[0]) {
    const size_t sm = short_smem(pl->Q, pl->slot_n);
    int occ_short = 0;
    const ShortVariant &sv = pick_short(pl->Q, pl->slot_n);
    for (PullFn f : {sv.words[0], sv.words[1], sv.words[2], sv.slots[1], sv.slots[2]}) {
      // the limit is the kernel's, which plans of other widths share: that of the widest rows
      if (sm > 48 * 1024)
        cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)short_smem(SHORT_MAX_Q, slot_entries(2 * SHORT_MAX_Q)));
      occ_short = std::max(occ_short, occupancy_grid(f, SH_WARPS * 32, sm, 8));
    }
    const uint64_t stasks = pl->npieces + ((uint64_t)V + short_tile(pl->Q) - 1) / short_tile(pl->Q);
    pl->grid_short = (int)std::max<uint64_t>(1, std::min<uint64_t>(occ_short, (stasks + SH_WARPS - 1) / SH_WARPS));
  }
  pl->grid_sparse = occupancy_grid(k_sparse, 256, 0, 8);
  pl->grid_push = occupancy_grid(k_push, 256, 0, 8);
  pl->grid_v = sm_count() * 8;
  *out = pl;
  return VS_OK;
}

// Device bytes vs_expand_plan_create allocates for these arguments (the
// serving loop admits queries by this number).
int vs_expand_plan_footprint(const vs_graph *g, uint32_t S, const vs_expand_params *p, uint64_t *bytes) {
  if (!g || !p || !bytes) return fail(VS_ERR_ARG, "null argument");
  const uint64_t V = g->V, W = words_per_col(S);
  const bool use_vis = p->path_type != VS_PATH_ANY;
  const bool use_acc = needs_acc(*p);
  uint64_t cap = p->pair_capacity ? p->pair_capacity
                                  : std::max<uint64_t>(1u << 20, std::min<uint64_t>((uint64_t)S * V / 8, 1ull << 25));
  cap = std::max<uint64_t>(cap, S);
  uint64_t b = (2 + use_vis + use_acc) * V * W * 8;             // frontier pair, visited, accumulator
  b += 5 * V * 4;                                                 // flags x2, resflag, push list, touched
  // heavy targets: at most a piece per piece_edges entries and one per target, a row per two pieces
  const uint64_t list_edges = (p->direction == VS_DIR_BOTH && g->directed ? 2 : 1) * g->E;
  b += cap * (2 * 8 + 2 * 8 + 8) + ((cap + 1023) / 1024 + 1) * 8;  // pair lists, degrees, offsets, block sums
  b += (uint64_t)S * 4 * 3 + sizeof(Ctr) + (uint64_t)(p->k_max + 1) * W * 8;
  uint32_t qs = p->slice_words ? (p->slice_words + 1) / 2 : (uint32_t)(W / 2);
  qs = std::max<uint32_t>(1, std::min<uint32_t>(qs, 256));
  const uint32_t nslices = (uint32_t)((W / 2 + qs - 1) / qs);
  const int L = pick_variant(qs).L;
  const uint64_t thr = p->hub_threshold ? std::min(p->hub_threshold, HEAVY_MAX) : heavy_default(L);
  // (of two lists one each may already be two pieces, whatever their length)
  const bool two = p->direction == VS_DIR_BOTH && g->directed;
  const uint64_t multi = std::min<uint64_t>(V, list_edges / std::max<uint64_t>(1, std::max<uint64_t>(thr, two ? 0 : piece_edges(L))));
  b += 16 * (16 + list_edges / piece_edges(L) + 2 * std::min<uint64_t>(V, list_edges / std::max<uint64_t>(1, thr)));
  b += multi * (W * 8 + 4 + 4 * nslices) + (uint64_t)(p->k_max + 1) * (W * 8 + 4 * nslices);
  const bool slots = short_slots_ok(S, nslices, p->short_share, V, (uint32_t)W);
  if (bits_ok((uint32_t)V, qs, slots, list_edges)) b += bits_smem((uint32_t)V);
  if (slots)
    b += 2 * V * (2 * slot_entries((uint32_t)W) + sizeof(Tiny));  // short-row words and slots of both buffers
  *bytes = b;
  return VS_OK;
}

int vs_expand_plan_free(vs_expand_plan *plan) { return plan_free(plan); }

int vs_expand_plan_run(vs_expand_plan *pl, const uint32_t *sources, const uint32_t *targets,
                       int32_t *distances, vs_stream_t stream) {
  if (!pl || !sources) return fail(VS_ERR_ARG, "vs_expand_plan_run: null argument");
  const vs_expand_params &p = pl->p;
  if (p.path_type == VS_PATH_FIND_SHORTEST && (!targets || !distances))
    return fail(VS_ERR_ARG, "FindShortest needs targets and distances");
  cudaStream_t st = S(stream);
  if (st != pl->last_stream) {  // earlier work on the plan ran in another stream's order
    VS_CK(cudaStreamSynchronize(pl->last_stream));
    pl->last_stream = st;
  }
  const vs_graph *g = pl->g;
  const uint32_t V = g->V, S_ = pl->S, W = pl->W, Q = pl->Q;
  const size_t rowbytes = (size_t)V * W * 8;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  VS_CK(cudaStreamIsCapturing(st, &cap));
  const bool timing = pl->timing && cap == cudaStreamCaptureStatusNone;  // events are not captured
  VS_TRY(copy_in(pl->d_src, sources, S_, st));
  if (pl->d_tgt) VS_TRY(copy_in(pl->d_tgt, targets, S_, st));
  if (pl->acc && pl->vis) VS_CK(cudaMemsetAsync(pl->vis, 0, rowbytes, st));  // no row marks
  // run start: clean frontier buffers, zero counters, and the rows of the result
  // matrix (visited or accumulator) that the previous run marked in resflag
  { k_run_start<<<pl->grid_v, 256, 0, st>>>(
        reinterpret_cast<uint4 *>(pl->buf[0]), pl->flag[0], reinterpret_cast<uint4 *>(pl->buf[1]), pl->flag[1],
        reinterpret_cast<uint4 *>(pl->acc ? pl->acc : pl->vis), pl->resflag, V, Q, reinterpret_cast<uint4 *>(pl->ctr),
        (uint32_t)(pl->ctr_bytes / 16)); vs::note_launch(); }
  const Lists in = pull_lists(g, p.direction), outl = push_lists(g, p.direction);
  SeedArgs sa;
  sa.sources = pl->d_src;
  sa.S = S_;
  sa.W = W;
  sa.buf0 = pl->buf[0];
  sa.flag0 = pl->flag[0];
  sa.vis = pl->vis;
  sa.acc = (pl->use_acc && p.k_min == 0) ? pl->acc : nullptr;
  sa.pairs0 = pl->pairs[0];
  sa.pdeg0 = pl->pdeg[0];
  sa.resflag = pl->resflag;
  sa.res_vis = pl->use_vis && !pl->use_acc;
  sa.out = outl;
  sa.ctr = pl->ctr;
  sa.V = V;
  sa.multislice = pl->nslices > 1;
  sa.rowk = pl->use_hmask ? pl->rowk : nullptr;
  sa.stats = pl->collect_stats || pl->log_features || (pl->picker && p.use_picker);
  vs::launch_next(k_seed, std::max(1u, std::min((S_ + 255) / 256, (uint32_t)sm_count() * 4)), 256, 0, st, sa);
  VS_CK(cudaGetLastError());
  if (pl->layer_out[0])
    vs::launch_next(k_copy_layer, pl->grid_v, 256, 0, st, reinterpret_cast<const uint4 *>(pl->buf[0]), pl->flag[0],
                                             reinterpret_cast<uint4 *>(pl->layer_out[0]), V, Q, pl->ctr, 0);
  if (p.path_type == VS_PATH_FIND_SHORTEST)
    vs::launch_next(k_dist_init, std::max(1u, std::min((S_ + 255) / 256, 1024u)), 256, 0, st, pl->d_src, pl->d_tgt,
                                                                              pl->d_dist, S_, V, pl->ctr);
  const PullVariant &var = pick_variant(pl->qslice);
  const int forced = p.strategy == VS_STRAT_PULL ? ST_PULL
                     : p.strategy == VS_STRAT_PUSH ? ST_PUSH
                     : p.strategy == VS_STRAT_SPARSE ? ST_SPARSE
                                                     : 0;
  // a PULL hop may leave the short rows of its layer in their slots when the
  // layer has a successor and nothing reads its rows directly (FindShortest
  // checks every layer's rows; a kept layer is copied out)
  auto leave_in_slots = [&](uint32_t hh) {
    return pl->slot[0] != nullptr && hh >= 1 && hh < p.k_max && p.path_type != VS_PATH_FIND_SHORTEST &&
           pl->layer_out[hh] == nullptr;
  };
  // a Shortest SPARSE hop leaves its layer's rows in its pair list when a
  // later hop may build them (not the last hop, not an exported layer, not
  // FindShortest, whose target check reads every layer's rows) and the plan
  // has a short-row index (without one every PULL hop reads whole rows, so
  // building them later only adds a pass)
  auto defer_rows = [&](uint32_t hh) {
    return pl->use_vis && pl->slot[0] != nullptr && hh >= 1 && hh < p.k_max &&
           p.path_type != VS_PATH_FIND_SHORTEST && !pl->layer_out[hh];
  };
  // PUSH runs only when forced (for the run or a hop) or enabled in the
  // fixed planner (push_frac > 0)
  bool any_forced_push = forced == ST_PUSH;
  for (uint32_t hh = 1; hh <= p.k_max; hh++) any_forced_push |= pl->hop_forced[hh] == ST_PUSH;
  // (the picker chooses PUSH only where the plan enables it)
  const bool can_push = any_forced_push || pl->push_frac > 0;
  const bool stats = pl->collect_stats || pl->log_features || (pl->picker && p.use_picker);
  for (uint32_t h = 1; h <= p.k_max; h++) {
    const int fb = (h - 1) & 1, nbuf = h & 1;
    const bool acc_on = pl->use_acc && h >= p.k_min && h <= p.k_max;
    DecideArgs da;
    da.ctr = pl->ctr;
    da.h = h;
    da.path = p.path_type;
    da.S = S_;
    da.V = V;
    da.E = g->E;
    da.forced = pl->hop_forced[h] ? pl->hop_forced[h] : forced;
    da.log_features = pl->log_features;
    da.both = p.direction == VS_DIR_BOTH && g->directed;
    da.pair_cap = pl->pair_cap;
    da.bits_ok = pl->bits != nullptr;
    da.sparse_frac = pl->sparse_frac;
    da.push_frac = pl->push_frac;
    da.picker = pl->picker;
    da.picker_on = p.use_picker;
    da.push_ok = can_push;
    da.rowk = pl->use_hmask ? pl->rowk : nullptr;
    da.short_min = pl->short_min;
    da.last = h == p.k_max && pl->use_vis && !pl->use_acc && p.path_type != VS_PATH_FIND_SHORTEST && !pl->layer_out[h];
    da.gen = !da.last && (acc_on || !leave_in_slots(h));
    da.W = W;
    da.k_min = p.k_min;
    da.k_max = p.k_max;
    // the seed and SPARSE hops count their layer's statistics; after a PULL or
    // PUSH hop only a picker that may choose PUSH (or logging) needs the pass
    const bool picker_only = !pl->collect_stats && !pl->log_features;
    if (stats && h > 1 && !(picker_only && !can_push))
      vs::launch_next(k_hop_stats, pl->grid_v, 256, 0, st, pl->flag[fb], outl, V, pl->ctr, h, picker_only, can_push);
    vs::launch_next(k_decide, 1, 256, 0, st, da);
    // hop_ms covers what the chosen strategy costs, not the statistics and decision before it
    if (timing) cudaEventRecord(pl->ev[3 * h], st);
    PrepArgs prep;
    prep.pairs = pl->pairs[fb];
    prep.cnt = pl->touched;
    prep.F = reinterpret_cast<unsigned long long *>(pl->buf[fb]);
    prep.flagF = pl->flag[fb];
    prep.N = reinterpret_cast<uint4 *>(pl->buf[nbuf]);
    prep.flagN = pl->flag[nbuf];
    prep.tiny = pl->tiny[fb];
    prep.slots = pl->slot[fb];
    prep.bits = pl->bits;
    prep.V = V;
    prep.W = W;
    prep.Q = Q;
    prep.slot_n = pl->slot_n;
    prep.cap = pl->pair_cap;
    prep.ctr = pl->ctr;
    prep.h = h;
    prep.deferred = defer_rows(h - 1);
    prep.virt = pl->slot[0] && leave_in_slots(h - 1);
    prep.clear = h > 1;  // hop 1 writes a buffer the run start cleared
    if (h > 1 || pl->slot[0]) vs::launch_next(k_hop_prep, pl->grid_v, 256, 0, st, prep);
    SparseArgs sp;
    sp.ctr = pl->ctr;
    sp.h = h;
    sp.resflag = pl->resflag;
    sp.res_vis = pl->use_vis && !pl->use_acc;
    sp.hmask = pl->use_hmask ? reinterpret_cast<const unsigned long long *>(pl->hmask + (size_t)h * W) : nullptr;
    sp.pin = pl->pairs[fb];
    sp.pout = pl->pairs[nbuf];
    sp.cap = pl->pair_cap;
    sp.out = outl;
    sp.W = W;
    sp.N = reinterpret_cast<unsigned long long *>(pl->buf[nbuf]);
    sp.vis = reinterpret_cast<unsigned long long *>(pl->vis);
    sp.acc = reinterpret_cast<unsigned long long *>(pl->acc);
    sp.flagN = pl->flag[nbuf];
    sp.shortest = pl->use_vis;
    sp.acc_on = acc_on;
    sp.doff = pl->doff;
    sp.pdeg_out = pl->pdeg[nbuf];
    sp.stats = stats && h < p.k_max;
    sp.last = h == p.k_max && pl->use_vis && p.path_type != VS_PATH_FIND_SHORTEST && !pl->layer_out[h];
    sp.defer = defer_rows(h);
    sp.bsum = pl->bsum;
    vs::launch_next(k_pscan, pl->grid_v, 256, 0, st, pl->pdeg[fb], pl->doff, pl->bsum, pl->ctr, h, pl->pair_cap);
    vs::launch_next(k_sparse, pl->grid_sparse, 256, 0, st, sp);
    PushArgs pa;
    pa.ctr = pl->ctr;
    pa.h = h;
    pa.resflag = pl->resflag;
    pa.res_vis = pl->use_vis && !pl->use_acc;
    pa.hmask = pl->use_hmask ? reinterpret_cast<const unsigned long long *>(pl->hmask + (size_t)h * W) : nullptr;
    pa.out = outl;
    pa.F = reinterpret_cast<const unsigned long long *>(pl->buf[fb]);
    pa.N = reinterpret_cast<unsigned long long *>(pl->buf[nbuf]);
    pa.vis = reinterpret_cast<unsigned long long *>(pl->vis);
    pa.acc = reinterpret_cast<unsigned long long *>(pl->acc);
    pa.flagN = pl->flag[nbuf];
    pa.active = pl->push_list;
    pa.touched = pl->touched;
    pa.W = W;
    pa.shortest = pl->use_vis;
    pa.acc_on = acc_on;
    if (can_push) {  // PUSH kernels only when the hop can run PUSH
      vs::launch_next(k_push_reset, 1, 1, 0, st, pl->ctr);
      vs::launch_next(k_push_compact, pl->grid_v, 256, 0, st, pl->flag[fb], V, pl->push_list, pl->ctr, h);
      vs::launch_next(k_push, pl->grid_push, 256, 0, st, pa);
      vs::launch_next(k_push_epilogue, pl->grid_push, 256, 0, st, pa);
    }
    PullArgs a;
    a.resflag = pl->resflag;
    a.res_vis = pl->use_vis && !pl->use_acc;
    a.hmask = pl->use_hmask ? reinterpret_cast<const uint4 *>(pl->hmask + (size_t)h * W) : nullptr;
    a.in = in;
    a.F = reinterpret_cast<const uint4 *>(pl->buf[fb]);
    a.N = reinterpret_cast<uint4 *>(pl->buf[nbuf]);
    a.vis = reinterpret_cast<uint4 *>(pl->vis);
    a.acc = reinterpret_cast<uint4 *>(pl->acc);
    a.flagF = pl->flag[fb];
    a.flagN = pl->flag[nbuf];
    a.V = V;
    a.Q = Q;
    a.qslice = pl->qslice;
    a.multislice = pl->nslices > 1;
    a.shortest = pl->use_vis;
    a.acc_on = acc_on;
    // the last hop's layer is read by nothing when the result is the visited
    // matrix or the accumulator (FindShortest checks every layer's targets)
    a.last = h == p.k_max && (pl->use_vis || pl->use_acc) && p.path_type != VS_PATH_FIND_SHORTEST &&
             !pl->layer_out[h];
    a.heavy_threshold = pl->nheavy ? pl->heavy_threshold : 0;
    a.pieces = pl->pieces;
    a.npieces = pl->npieces;
    a.piece_edges = piece_edges(var.L);
    a.heavy_np = pl->heavy_np;
    a.heavy_left = pl->heavy_left;
    a.heavy_rows = pl->heavy_rows;
    a.tile = pl->tile;
    a.queue = pl->queue + (size_t)h * pl->nslices;
    a.Uin = pl->un + (size_t)(h - 1) * Q;
    a.Uout = pl->un + (size_t)h * Q;
    a.S = S_;
    a.ctr = pl->ctr;
    a.h = h;
    const bool keep_short = pl->slot[0] && h < p.k_max && !a.last;  // the next hop may read this layer's words
    a.virt_out = keep_short && leave_in_slots(h);
    a.tiny_in = pl->slot[0] ? pl->tiny[fb] : nullptr;
    a.slot_in = pl->slot[0] ? reinterpret_cast<const uint4 *>(pl->slot[fb]) : nullptr;
    a.tiny_out = keep_short ? pl->tiny[nbuf] : nullptr;
    a.slot_out = keep_short ? pl->slot[nbuf] : nullptr;
    a.slot_n = pl->slot_n;
    a.out = outl;
    short_layout(a, short_tile(Q));
    if (timing) cudaEventRecord(pl->ev[3 * h + 1], st);
    if (pl->slot[0]) {  // words and slots of a layer SPARSE, PUSH or the seed wrote, when this hop reads them
      vs::launch_next(k_pairs_slots, pl->grid_v, 256, 0, st, pl->pairs[fb], pl->touched, pl->slot[fb], pl->slot_n, pl->pair_cap,
                                                pl->ctr, h);
      vs::launch_next(k_short_index, pl->grid_v, 256, 0, st, prep);
    }
    a.bits = pl->bits;
    if (pl->bits && h > 1) vs::launch_next(var.bits, dim3(pl->grid_bits, pl->nslices), 1024, bits_smem(V), st, a);
    vs::launch_next(var.pull, dim3(pl->grid_pull, pl->nslices), 256, 0, st, a);
    if (pl->slot[0]) {
      const ShortVariant &sv = pick_short(Q, pl->slot_n);
      const size_t sm = short_smem(Q, pl->slot_n);
      const bool last = a.last && a.shortest && !a.acc_on;
      a.list_too = !last && a.tiny_out && a.virt_out && !a.acc_on;
      if (a.list_too) vs::launch_next(sv.words[SH_LIST], pl->grid_short, SH_WARPS * 32, sm, st, a);
      vs::launch_next(sv.words[last ? SH_LAST : SH_GEN], pl->grid_short, SH_WARPS * 32, sm, st, a);
      a.list_too = 0;
      vs::launch_next(sv.slots[last ? SH_LAST : SH_GEN], pl->grid_short, SH_WARPS * 32, sm, st, a);
    }
    if (p.path_type == VS_PATH_FIND_SHORTEST)
      vs::launch_next(k_find_check, std::max(1u, std::min((S_ + 255) / 256, 1024u)), 256, 0, st,
          pl->buf[nbuf], pl->d_tgt, pl->d_dist, S_, W, V, pl->ctr, h);
    if (pl->layer_out[h])
      vs::launch_next(k_copy_layer, pl->grid_v, 256, 0, st, reinterpret_cast<const uint4 *>(pl->buf[nbuf]), pl->flag[nbuf],
                                               reinterpret_cast<uint4 *>(pl->layer_out[h]), V, Q, pl->ctr, h);
    if (timing) cudaEventRecord(pl->ev[3 * h + 2], st);
    VS_CK(cudaGetLastError());
  }
  pl->timed_hops = timing ? p.k_max : 0;
  if (pl->clear_diag)
    vs::launch_next(k_clear_diag, std::max(1u, std::min((S_ + 255) / 256, 1024u)), 256, 0, st, pl->vis, pl->d_src,
                                                                                S_, W, V);
  if (p.path_type == VS_PATH_FIND_SHORTEST)
    VS_TRY(copy_in(distances, (const int32_t *)pl->d_dist, S_, st));
  VS_CK(cudaGetLastError());
  // result view
  vs_bitmat &r = pl->result;
  r = vs_bitmat{};
  r.rows = S_;
  r.cols = V;
  r.wpc = W;
  r.kind = VS_KIND_VARROW;
  const int lb = p.k_max & 1;  // buffer of layer k_max (the result of Any [k, k])
  r.words = pl->use_acc ? pl->acc : pl->use_vis ? pl->vis : pl->buf[lb];
  r.row_map = pl->d_src;
  r.col_map = nullptr;
  r.colnz = (pl->use_acc || pl->use_vis) ? pl->resflag : pl->flag[lb];
  r.owns_words = false;
  r.view = true;
  pl->has_result = p.path_type != VS_PATH_FIND_SHORTEST;
  return VS_OK;
}

int vs_expand_plan_result(vs_expand_plan *pl, vs_bitmat **view) {
  if (!pl || !view) return fail(VS_ERR_ARG, "null argument");
  if (!pl->has_result) return fail(VS_ERR_ARG, "plan has no matrix result");
  vs_bitmat *m = new vs_bitmat(pl->result);
  m->view = true;
  *view = m;
  return VS_OK;
}

int vs_expand_plan_stats(vs_expand_plan *pl, vs_expand_stats *stats, vs_stream_t stream) {
  if (!pl || !stats) return fail(VS_ERR_ARG, "null argument");
  Ctr h;
  VS_CK(cudaMemcpyAsync(&h, pl->ctr, sizeof(Ctr), cudaMemcpyDeviceToHost, S(stream)));
  VS_CK(cudaStreamSynchronize(S(stream)));
  std::memset(stats, 0, sizeof(*stats));
  if (h.error & 2) return fail(VS_ERR_ARG, "a row hop limit set on the device exceeds k_max %u", pl->p.k_max);
  if (h.error) return fail(VS_ERR_ARG, "a source or target vertex id is >= V (%u)", pl->g->V);
  stats->hops_run = (uint32_t)h.hops_run;
  stats->found = (uint32_t)h.found;
  uint64_t vc = pl->S;
  for (int i = 0; i <= VS_MAX_HOPS; i++) {
    stats->new_bits[i] = h.hop[i].new_bits;
    stats->active_vertices[i] = h.hop[i].active_vertices;
    stats->active_edges[i] = h.hop[i].active_edges;
    stats->pairs[i] = h.hop[i].pairs;
    stats->strategy[i] = h.hop[i].strategy;
    stats->short_pull[i] = h.hop[i].short_pull ? (h.hop[i].short_slots ? 2 : 1) : 0;
    stats->short_rows[i] = h.hop[i].short_rows & 0xFFFFFFFFull;
    stats->tiny_rows[i] = h.hop[i].short_rows >> 32;
    stats->short_edges[i] = h.hop[i].short_edges;
    if (i >= 1 && i <= h.hops_run) vc += h.hop[i].new_bits;
  }
  for (uint32_t i = 1; i <= pl->timed_hops && i <= VS_MAX_HOPS; i++) {
    float a = 0, b = 0;
    if (cudaEventElapsedTime(&a, pl->ev[3 * i], pl->ev[3 * i + 2]) == cudaSuccess) stats->hop_ms[i] = a;
    if (cudaEventElapsedTime(&b, pl->ev[3 * i + 1], pl->ev[3 * i + 2]) == cudaSuccess) stats->pull_ms[i] = b;
  }
  stats->visit_count = pl->use_vis ? vc : 0;
  return VS_OK;
}

int vs_expand_plan_set_tuning(vs_expand_plan *pl, double sparse_frac, double push_frac,
                              int collect_stats, int timing) {
  if (!pl) return fail(VS_ERR_ARG, "null plan");
  if (sparse_frac >= 0) pl->sparse_frac = sparse_frac;
  if (push_frac >= 0) pl->push_frac = push_frac;
  pl->collect_stats = collect_stats != 0;
  if (timing && !pl->timing) {
    for (cudaEvent_t &e : pl->ev)
      if (!e) VS_CK(cudaEventCreate(&e));
  }
  pl->timing = timing != 0;
  return VS_OK;
}

int vs_expand_plan_set_picker(vs_expand_plan *pl, const vs_picker *p) {
  if (!pl) return fail(VS_ERR_ARG, "null plan");
  pl->picker = p ? vs_picker_device_weights(p) : nullptr;
  return VS_OK;
}

int vs_expand_plan_set_hop_strategies(vs_expand_plan *pl, const int32_t *strategies, uint32_t n) {
  if (!pl) return fail(VS_ERR_ARG, "null plan");
  for (int h = 0; h <= VS_MAX_HOPS; h++) pl->hop_forced[h] = 0;
  for (uint32_t h = 1; strategies && h < n && h <= VS_MAX_HOPS; h++) {
    const int s = strategies[h];
    if (s < VS_STRAT_AUTO || s > VS_STRAT_SPARSE) return fail(VS_ERR_ARG, "unknown strategy %d", s);
    pl->hop_forced[h] = s == VS_STRAT_PULL ? ST_PULL : s == VS_STRAT_PUSH ? ST_PUSH : s == VS_STRAT_SPARSE ? ST_SPARSE : 0;
  }
  return VS_OK;
}

// Batched queries: row i of the plan belongs to a query whose hop range ends
// at row_kmax[i] (<= the plan's k_max).  Rows stop growing after their own
// last hop, so every query's rows equal the result of running it alone.
int vs_expand_plan_set_row_limits(vs_expand_plan *pl, const uint8_t *row_kmax, uint32_t n) {
  if (!pl) return fail(VS_ERR_ARG, "null plan");
  if (!row_kmax) {
    pl->use_hmask = false;
    return VS_OK;
  }
  if (n != pl->S) return fail(VS_ERR_ARG, "row limits need one entry per source row (%u)", pl->S);
  const uint32_t K = pl->p.k_max, W = pl->W;
  std::vector<uint64_t> m((size_t)(K + 1) * W, 0);
  bool all = true;
  uint32_t rk[2] = {0, 0};
  for (uint32_t i = 0; i < n; i++) {
    if (row_kmax[i] > K) return fail(VS_ERR_ARG, "row %u hop limit %u exceeds k_max %u", i, row_kmax[i], K);
    all &= row_kmax[i] == K;
    rk[0] = std::max<uint32_t>(rk[0], row_kmax[i]);
    for (uint32_t h = 1; h <= row_kmax[i]; h++) m[(size_t)h * W + i / 64] |= 1ull << (i % 64);
  }
  if (!all && !pl->use_acc && !pl->use_vis)
    return fail(VS_ERR_UNSUPPORTED, "row limits need an accumulating plan (Any with k_min < k_max, or Shortest)");
  // the mask is written even when unused, so a run captured with limits stays right
  VS_CK(cudaStreamSynchronize(pl->last_stream));  // no earlier run still reads the mask
  VS_CK(cudaMemcpy(pl->hmask, m.data(), 8 * m.size(), cudaMemcpyHostToDevice));
  VS_CK(cudaMemcpy(pl->rowk, rk, sizeof(rk), cudaMemcpyHostToDevice));
  pl->use_hmask = !all;
  return VS_OK;
}

// Row limits from a device array, stream-ordered (capturable): the mask of
// every hop is built by k_row_mask; rows at index >= n get limit 0 (they
// never grow).  A limit above k_max is clamped and reported as VS_ERR_ARG by
// the next run.
int vs_expand_plan_set_row_limits_device(vs_expand_plan *pl, const uint8_t *row_kmax, uint32_t n,
                                         vs_stream_t stream) {
  if (!pl || !row_kmax) return fail(VS_ERR_ARG, "vs_expand_plan_set_row_limits_device: null argument");
  if (n > pl->S) return fail(VS_ERR_ARG, "%u row limits for a plan of %u rows", n, pl->S);
  if (!pl->use_acc && !pl->use_vis)
    return fail(VS_ERR_UNSUPPORTED, "row limits need an accumulating plan (Any with k_min < k_max, or Shortest)");
  cudaStream_t st = S(stream);
  if (st != pl->last_stream) {
    VS_CK(cudaStreamSynchronize(pl->last_stream));
    pl->last_stream = st;
  }
  VS_CK(cudaMemsetAsync(pl->rowk, 0, 2 * sizeof(uint32_t), st));
  const uint32_t W = pl->W;
  { k_row_mask<<<(W + 7) / 8, 256, 0, st>>>(row_kmax, n, pl->p.k_max, W, pl->hmask, pl->rowk); vs::note_launch(); }
  VS_CK(cudaGetLastError());
  pl->use_hmask = true;
  return VS_OK;
}

// Kernel shape of the PULL hops: the shapes it chose from are gone (the kernels
// run one shape per row width); the kind is still taken, so saved settings stay
// valid.
int vs_expand_plan_set_pull_kernel(vs_expand_plan *pl, int kind) {
  if (!pl || kind < 0 || kind > 7) return fail(VS_ERR_ARG, "pull kernel variant must be 0..7");
  return VS_OK;
}

int vs_expand_plan_log_features(vs_expand_plan *pl, int on) {
  if (!pl) return fail(VS_ERR_ARG, "null plan");
  pl->log_features = on != 0;
  return VS_OK;
}

int vs_expand_plan_features(vs_expand_plan *pl, float *features, vs_stream_t stream) {
  if (!pl || !features) return fail(VS_ERR_ARG, "null argument");
  VS_CK(cudaMemcpyAsync(features, pl->ctr->feat, sizeof(float) * 32 * (VS_MAX_HOPS + 1), cudaMemcpyDefault,
                        S(stream)));
  VS_CK(cudaStreamSynchronize(S(stream)));
  return VS_OK;
}

// VExpand with_distance, Dense strategy (copy_to_multi_MT, vexpand.cpp:356-378):
// layers k_min..k_actual each as a VarRow matrix with the sources as row map.
int vs_expand_layers(vs_graph *g, const uint32_t *sources, uint32_t S, const vs_expand_params *p,
                     vs_bitmat **layers, uint32_t *nlayers, vs_stream_t stream) {
  if (!g || !p || !layers || !nlayers) return fail(VS_ERR_ARG, "vs_expand_layers: null argument");
  if (p->path_type == VS_PATH_FIND_SHORTEST)
    return fail(VS_ERR_ARG, "FindShortest reports distances per pair, not layers");
  if (p->k_min > p->k_max || p->k_max > VS_MAX_HOPS) return fail(VS_ERR_ARG, "bad hop range [%u, %u]", p->k_min, p->k_max);
  const uint32_t n = p->k_max - p->k_min + 1;
  *nlayers = 0;
  for (uint32_t i = 0; i < n; i++) layers[i] = nullptr;
  if (S == 0) return VS_OK;  // no start vertex: no layer (VExpand::before_execution)
  cudaStream_t st = vs::S(stream);
  vs_expand_plan *pl = nullptr;
  VS_TRY(vs_expand_plan_create(g, S, p, &pl));
  pl->collect_stats = true;
  int rc = VS_OK;
  for (uint32_t i = 0; i < n && rc == VS_OK; i++) {
    rc = bitmat_alloc(S, g->V, VS_KIND_VARROW, st, &layers[i]);
    if (rc == VS_OK) {
      pl->layer_out[p->k_min + i] = layers[i]->words;
      rc = vs_bitmat_set_maps(layers[i], sources, nullptr, stream);
    }
  }
  if (rc == VS_OK) {
    const cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) rc = cuda_fail(e, "vs_expand_layers", __FILE__, __LINE__);
  }
  if (rc == VS_OK) rc = vs_expand_plan_run(pl, sources, nullptr, nullptr, stream);
  vs_expand_stats stt{};
  if (rc == VS_OK) rc = vs_expand_plan_stats(pl, &stt, stream);
  plan_free(pl);
  uint32_t keep = 0;
  if (rc == VS_OK) {
    const uint32_t k_actual = stt.hops_run;  // last hop run (VExpand::after_child, vexpand.cpp:223)
    keep = k_actual >= p->k_min ? std::min(k_actual, p->k_max) - p->k_min + 1 : 0;
  }
  for (uint32_t i = keep; i < n; i++) {
    vs_bitmat_free(layers[i]);
    layers[i] = nullptr;
  }
  *nlayers = keep;
  return rc;
}

int vs_expand(vs_graph *g, const uint32_t *sources, uint32_t S, const vs_expand_params *p,
              const uint32_t *targets, int32_t *distances, vs_bitmat **out, vs_expand_stats *stats,
              vs_stream_t stream) {
  if (!g || !p) return fail(VS_ERR_ARG, "vs_expand: null argument");
  if (S == 0) {
    // VExpand::before_execution returns false on an empty start list: empty result
    if (out && p->path_type != VS_PATH_FIND_SHORTEST)
      return bitmat_alloc(0, g->V, VS_KIND_VARROW, vs::S(stream), out);
    if (stats) std::memset(stats, 0, sizeof(*stats));
    return VS_OK;
  }
  cudaStream_t st = vs::S(stream);
  vs_expand_plan *pl = plan_cache_take(g, S, *p);
  if (pl) {
    if (pl->cache_ev) VS_CK(cudaStreamWaitEvent(st, pl->cache_ev, 0));
  } else {
    int rc0 = vs_expand_plan_create(g, S, p, &pl);
    if (rc0 == VS_ERR_OOM) {  // the cached plans may hold the memory: release them and retry once
      vs_release_cached();
      rc0 = vs_expand_plan_create(g, S, p, &pl);
    }
    if (rc0 != VS_OK) return rc0;
    pl->key = *p;
    pl->graph_serial = g->serial;
    vs_expand_plan_footprint(g, S, p, &pl->bytes);
  }
  pl->collect_stats = stats != nullptr;
  int rc = vs_expand_plan_run(pl, sources, targets, distances, stream);
  if (rc == VS_OK && stats) rc = vs_expand_plan_stats(pl, stats, stream);
  if (rc == VS_OK && !stats) {
    int err = 0;
    cudaError_t e = cudaMemcpyAsync(&err, &pl->ctr->error, sizeof(int), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess)
      rc = cuda_fail(e, "vs_expand", __FILE__, __LINE__);
    else if (err)
      rc = fail(VS_ERR_ARG, "a source or target vertex id is >= V (%u)", g->V);
  }
  if (rc != VS_OK) {  // a failed run leaves the plan out of the cache
    plan_free(pl);
    return rc;
  }
  if (out && p->path_type != VS_PATH_FIND_SHORTEST) {
    // the result is the plan's own result matrix, lent until the handle is freed
    vs_bitmat *m = new vs_bitmat(pl->result);
    m->view = true;
    m->owns_words = false;
    m->pool_plan = pl;
    m->st = st;
    *out = m;
    return VS_OK;
  }
  plan_cache_return(pl, st);
  return VS_OK;
}

int vs_release_cached(void) {
  std::vector<vs_expand_plan *> drop;
  {
    PlanCache &c = plan_cache();
    std::lock_guard<std::mutex> lk(c.mu);
    drop.swap(c.idle);
  }
  for (vs_expand_plan *d : drop) plan_free(d);
  return VS_OK;
}

}  // extern "C"
