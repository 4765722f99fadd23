// Mixture-of-experts routing and expert-parallel token exchange over NVLink peer memory.
//
// What the reference does with library calls and host round trips (softmax / topk,
// parallel/parallel_ep.py: argsort, bincount, a count all-to-all whose result is read on the host,
// a variable-size all-to-all, index_copy_, a weighted sum) is done here by five kernels, none of
// which returns anything to the host:
//
//   moe_router_kernel    gate GEMM (E is tiny: one warp per token, fp32 dot products), softmax,
//                        top-k, and for every (token, slot) copy its rank among the copies of the
//                        same expert inside the same 32-token block, plus per-block histograms
//   moe_plan_kernel      one CTA: prefix sums over the blocks, this rank's per-expert counts stored
//                        into every peer's count table (flag per source rank), then, from the full
//                        [ranks x experts] table, the row in the owner's buffer where this rank's
//                        copies of every expert start, the layout of the local expert segments
//                        (each starts on a multiple of 128 rows) and the load-balance loss
//   moe_push_kernel      dispatch (and the backward of combine): every copy's row is stored, scaled
//                        if asked, straight into the expert owner's buffer with 16-byte peer stores;
//                        every CTA counts itself in each destination's arrival word when its stores
//                        are fenced; the owner zeroes the padding rows of its segments
//   moe_pull_kernel      combine (and the backward of dispatch): a token's k expert outputs are read
//                        from their owners with 16-byte peer loads, weighted and summed; the same
//                        pass can produce the dot products that are the router-weight gradients
//   moe_router_bwd_kernel  softmax backward, dx = dlogits . Wg, dWg += dlogits^T x
//
// The expert GEMMs between push and pull (lb_gemm_ragged_epi, gemm_grouped.cu), whose epilogues are the activation and its backward, take the
// segment offsets and counts from device memory; the first of each direction waits for the arrival word itself.
//
// All waits on a peer are bounded (comm.cuh) and report through lb_moe_status(); row indices are
// checked against the buffer capacity before every store or load (a routing so skewed that a rank
// would receive more than its capacity sets the status word instead of writing out of bounds).
#include "comm.cuh"

static __device__ unsigned int g_moe_status[4] = {0, 0, 0, 0};

namespace {

constexpr int MOE_MAX_RANKS = 8;
constexpr int MOE_MAX_EXPERTS = 64;
constexpr int MOE_MAX_TOPK = 8;
constexpr int ROUTER_TOKENS = 32;       // tokens per router block (the unit of the within-block ranks)
constexpr int ROUTER_THREADS = 256;

// A copy routed to a row beyond the expert-side capacity is DROPPED (not dispatched, contributes
// nothing to the combine), as in capacity-factor routing; it is counted, not treated as a failure:
// word 2 = dropped copies / overfull plans since the last read, word 3 = largest row count asked for.
__device__ __forceinline__ void moe_overflow(unsigned rows_wanted) {
  atomicAdd(&g_moe_status[2], 1u);
  atomicMax(&g_moe_status[3], rows_wanted);
}
__device__ __forceinline__ void moe_fail(unsigned code, unsigned where) {
  if (atomicCAS(&g_moe_status[0], 0u, code) == 0u) atomicExch(&g_moe_status[1], where);
}

// -------------------------------------------------------------------------------------------
// Router
// -------------------------------------------------------------------------------------------
// Latency bound.  IN tokens of a warp go through the gate weights together, 8 experts at a time; the IN row vectors and the 8 weight vectors of
// a step are all loaded before the first is used (behind a branch per expert each load was waited for by itself: T 4096, H 2048, inputs not in
// L2, E 8 47 us, now 25; E 64 284, now 96).  The sums of a token are the same for every IN.
template <int IN>
__global__ void __launch_bounds__(ROUTER_THREADS)
moe_router_kernel(const bf16* __restrict__ x, const bf16* __restrict__ wg, int T, int H, int E, int k,
                  float* __restrict__ probs, int* __restrict__ idx, float* __restrict__ wts, int* __restrict__ within,
                  int* __restrict__ blk_hist, float* __restrict__ blk_psum) {
  grid_go();
  grid_wait();
  __shared__ int s_eid[ROUTER_TOKENS * MOE_MAX_TOPK];
  __shared__ int s_hist[MOE_MAX_EXPERTS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t0 = blockIdx.x * ROUTER_TOKENS;
  for (int i = threadIdx.x; i < MOE_MAX_EXPERTS; i += blockDim.x) s_hist[i] = 0;
  for (int i = threadIdx.x; i < ROUTER_TOKENS * MOE_MAX_TOPK; i += blockDim.x) s_eid[i] = -1;
  __syncthreads();
  const int nvec = H >> 3;
  constexpr int TPW = ROUTER_TOKENS / (ROUTER_THREADS / 32), NW = ROUTER_THREADS / 32;
  for (int i0 = 0; i0 < TPW && t0 + warp + i0 * NW < T; i0 += IN) {      // IN tokens of the warp at a time
    // logits[e] for e = lane, lane + 32 end up in lg[0] / lg[1] (E <= 64)
    float lg[IN][2];
#pragma unroll
    for (int i = 0; i < IN; i++) lg[i][0] = lg[i][1] = -INFINITY;
    for (int e0 = 0; e0 < E; e0 += 8) {                     // 8 experts per pass over the rows
      float acc[IN][8];
#pragma unroll
      for (int i = 0; i < IN; i++)
#pragma unroll
        for (int j = 0; j < 8; j++) acc[i][j] = 0.f;
      const int ne = min(8, E - e0);
      for (int v = lane; v < nvec; v += 32) {
        uint4 xr[IN], wr[8];
#pragma unroll
        for (int i = 0; i < IN; i++) {
          const int t = t0 + warp + (i0 + i) * NW;
          xr[i] = t < T ? reinterpret_cast<const uint4*>(x + (size_t)t * H)[v] : make_uint4(0, 0, 0, 0);
        }
#pragma unroll
        for (int j = 0; j < 8; j++) wr[j] = __ldg(reinterpret_cast<const uint4*>(wg + (size_t)(e0 + min(j, ne - 1)) * H) + v);
        float xf[IN][8];
#pragma unroll
        for (int i = 0; i < IN; i++) unpack8(xr[i], xf[i]);
#pragma unroll
        for (int j = 0; j < 8; j++) {
          if (j < ne) {
            float wf[8];
            unpack8(wr[j], wf);
#pragma unroll
            for (int i = 0; i < IN; i++)
#pragma unroll
              for (int c = 0; c < 8; c++) acc[i][j] = fmaf(xf[i][c], wf[c], acc[i][j]);
          }
        }
      }
#pragma unroll
      for (int i = 0; i < IN; i++)
#pragma unroll
        for (int j = 0; j < 8; j++) {
          const float s = warp_sum(acc[i][j]);
          if (j < ne) {
            const int e = e0 + j;
            if ((e & 31) == lane) { if (e < 32) lg[i][0] = s; else lg[i][1] = s; }
          }
        }
    }
#pragma unroll
    for (int i = 0; i < IN; i++) {
      const int tl = warp + (i0 + i) * NW, t = t0 + tl;
      if (t >= T) break;                                   // warp-uniform
      const float lg0 = lg[i][0], lg1 = lg[i][1];
      // softmax over experts (fp32), every lane ends with its own probabilities
      const float mx = warp_max(fmaxf(lg0, lg1));
      const float ex0 = (lane < E) ? __expf(lg0 - mx) : 0.f;
      const float ex1 = (lane + 32 < E) ? __expf(lg1 - mx) : 0.f;
      const float inv = 1.f / warp_sum(ex0 + ex1);
      const float p0 = ex0 * inv, p1 = ex1 * inv;
      if (lane < E) probs[(size_t)t * E + lane] = p0;
      if (lane + 32 < E) probs[(size_t)t * E + lane + 32] = p1;
      // top-k: k rounds of arg-max (lowest index wins ties)
      float q0 = (lane < E) ? p0 : -1.f, q1 = (lane + 32 < E) ? p1 : -1.f;
      for (int s = 0; s < k; s++) {
        float best = fmaxf(q0, q1);
        int bi = (q0 >= q1) ? lane : lane + 32;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          const float ob = __shfl_xor_sync(0xffffffffu, best, o);
          const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
          if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
        }
        if (lane == 0) {
          idx[(size_t)t * k + s] = bi;
          wts[(size_t)t * k + s] = best;
          s_eid[tl * k + s] = bi;
        }
        if (bi == lane) q0 = -1.f;
        if (bi == lane + 32) q1 = -1.f;
      }
    }
  }
  __syncthreads();
  // rank of every copy among the block's earlier copies of the same expert, in (token, slot) order
  const int ncopies = ROUTER_TOKENS * k;
  for (int c = threadIdx.x; c < ncopies; c += blockDim.x) {
    const int e = s_eid[c];
    if (e < 0) continue;
    int r = 0;
    for (int j = 0; j < c; j++) r += (s_eid[j] == e);
    within[(size_t)t0 * k + c] = r;
    atomicAdd(&s_hist[e], 1);
  }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    // probability mass per expert over the block's tokens, summed in token order (deterministic)
    float ps = 0.f;
    for (int tl = 0; tl < ROUTER_TOKENS && t0 + tl < T; tl++) ps += probs[(size_t)(t0 + tl) * E + e];
    blk_hist[(size_t)blockIdx.x * E + e] = s_hist[e];
    blk_psum[(size_t)blockIdx.x * E + e] = ps;
  }
}

// -------------------------------------------------------------------------------------------
// Plan
// -------------------------------------------------------------------------------------------
struct PlanParams {
  const int* blk_hist;      // [nblk, E]
  const float* blk_psum;    // [nblk, E]
  int* blk_base;            // [nblk, E] out: copies of expert e in earlier blocks of this rank
  int* dst_row0;            // [E] out: row in the owner's buffer where this rank's copies of e start
  int* seg;                 // [2 * LE + 2] out: offsets[LE], counts[LE], padded end, total received
  float* frac;              // [E] out: fraction of this rank's copies routed to e
  float* aux;               // [1] out: load-balance loss E * sum_e frac_e * mean_t p_te
  int nblk, E, LE, n, me, T, k, cap;
  int* cnt_all[MOE_MAX_RANKS];          // rank r's count table [2][n][E]
  unsigned int* flags[MOE_MAX_RANKS];   // rank r's "counts arrived" words [n]
  int parity;
  unsigned int epoch;
  unsigned long long wait_ns;
};

__global__ void __launch_bounds__(256) moe_plan_kernel(const PlanParams p) {
  if (p.n == 1) grid_go();
  grid_wait();
  __shared__ int s_cnt[MOE_MAX_EXPERTS];
  __shared__ float s_ps[MOE_MAX_EXPERTS];
  __shared__ int s_all[MOE_MAX_RANKS * MOE_MAX_EXPERTS];
  __shared__ int s_fail;
  const int tid = threadIdx.x;
  if (tid == 0) s_fail = 0;
  // Copies per expert, and those of earlier blocks: a warp per expert, a lane per block.  (A thread per expert that went through the
  // blocks one after the other: 128 blocks, 8 experts 16 us, now 9.)
  const int lane = tid & 31;
  for (int e = tid >> 5; e < p.E; e += 8) {
    int run = 0;
    float ps = 0.f;
    for (int b0 = 0; b0 < p.nblk; b0 += 128) {
      int hist[4];
      float psum[4];
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int b = b0 + 32 * i + lane;
        hist[i] = b < p.nblk ? p.blk_hist[(size_t)b * p.E + e] : 0;
        psum[i] = b < p.nblk ? p.blk_psum[(size_t)b * p.E + e] : 0.f;
      }
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int b = b0 + 32 * i + lane;
        int upto = hist[i];                                // inclusive sum over the lanes
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int v = __shfl_up_sync(0xffffffffu, upto, o);
          if (lane >= o) upto += v;
        }
        if (b < p.nblk) p.blk_base[(size_t)b * p.E + e] = run + upto - hist[i];
        run += __shfl_sync(0xffffffffu, upto, 31);
        ps += psum[i];
      }
    }
    ps = warp_sum(ps);
    if (lane == 0) {
      s_cnt[e] = run;
      s_ps[e] = ps;
      p.frac[e] = (float)run / (float)((long long)p.T * p.k);
      for (int r = 0; r < p.n; r++) p.cnt_all[r][((size_t)p.parity * p.n + p.me) * p.E + e] = run;
    }
  }
  __syncthreads();
  if (tid < p.n) {
    __threadfence_system();
    lbcomm::st_release_sys(p.flags[tid] + p.me, p.epoch);
    if (!lbcomm::flag_wait_ge(p.flags[p.me] + tid, p.epoch, p.wait_ns)) { s_fail = 1; moe_fail(1u, 1u); }
  }
  __syncthreads();
  if (s_fail) {
    for (int i = tid; i < 2 * p.LE + 2; i += blockDim.x) p.seg[i] = 0;      // no rows
    return;
  }
  const volatile int* mine = p.cnt_all[p.me] + (size_t)p.parity * p.n * p.E;
  for (int i = tid; i < p.n * p.E; i += blockDim.x) s_all[i] = mine[i];
  __syncthreads();
  if (tid < p.E) {
    const int d = tid / p.LE, le = tid - d * p.LE;
    int base = 0;
    for (int j = 0; j < le; j++) {          // padded sizes of the owner's earlier local experts
      int tot = 0;
      for (int s = 0; s < p.n; s++) tot += s_all[s * p.E + d * p.LE + j];
      base += (tot + 127) & ~127;
    }
    int before = 0, tot = 0;
    for (int s = 0; s < p.n; s++) {
      const int c = s_all[s * p.E + tid];
      if (s < p.me) before += c;
      tot += c;
    }
    p.dst_row0[tid] = base + before;
    if (d == p.me) {
      p.seg[le] = base;
      p.seg[p.LE + le] = tot;
      if (le == p.LE - 1) {
        const int end = base + ((tot + 127) & ~127);
        p.seg[2 * p.LE] = end;
        if (end > p.cap) moe_overflow((unsigned)end);        // more rows routed here than the buffers hold: the excess is dropped
      }
    }
  }
  if (tid == 0) {
    int total = 0;
    for (int le = 0; le < p.LE; le++)
      for (int s = 0; s < p.n; s++) total += s_all[s * p.E + p.me * p.LE + le];
    p.seg[2 * p.LE + 1] = total;
    float a = 0.f;
    for (int e = 0; e < p.E; e++) a += ((float)s_cnt[e] / (float)((long long)p.T * p.k)) * (s_ps[e] / (float)p.T);
    p.aux[0] = a * (float)p.E;
  }
}

// -------------------------------------------------------------------------------------------
// Push: dst_owner[row(t, s)] = scale[t, s] * src[t]
// -------------------------------------------------------------------------------------------
struct PushParams {
  const bf16* src;          // [T, H]
  const float* scale;       // [T, k] or null
  const int* idx;           // [T, k] expert of every copy
  const int* within;        // [T, k]   (compute_rows)
  const int* blk_base;      // [nblk, E] (compute_rows)
  const int* dst_row0;      // [E]       (compute_rows)
  int* rows;                // [T, k]: written when compute_rows, read otherwise
  const int* seg;           // local segment table (for zeroing the padding rows of `own`)
  bf16* own;                // this rank's buffer (== dst[me])
  bf16* dst[MOE_MAX_RANKS];
  unsigned int* arrive[MOE_MAX_RANKS];   // rank r's arrival word for this buffer
  int T, H, E, LE, k, n, me, cap, compute_rows;
};

__global__ void __launch_bounds__(256) moe_push_kernel(const PushParams p) {
  if (p.n == 1) grid_go();
  grid_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
  const int nvec = p.H >> 3;
  // padding rows of the local segments: rows [off + cnt, off + round_up(cnt, 128)) become zero
  for (int le = 0; le < p.LE; le++) {
    const int off = p.seg[le], cnt = p.seg[p.LE + le];
    const int pad0 = off + cnt, pad1 = min(off + ((cnt + 127) & ~127), p.cap);
    for (int r = pad0 + blockIdx.x * wpb + warp; r < pad1; r += gridDim.x * wpb) {
      uint4* d = reinterpret_cast<uint4*>(p.own + (size_t)r * p.H);
      for (int v = lane; v < nvec; v += 32) d[v] = make_uint4(0, 0, 0, 0);
    }
  }
  for (int t = blockIdx.x * wpb + warp; t < p.T; t += gridDim.x * wpb) {
    const uint4* sr = reinterpret_cast<const uint4*>(p.src + (size_t)t * p.H);
    uint4* drow[MOE_MAX_TOPK];
    float sc[MOE_MAX_TOPK];
#pragma unroll
    for (int s = 0; s < MOE_MAX_TOPK; s++) {
      drow[s] = nullptr;
      sc[s] = 1.f;
      if (s < p.k) {
        const int e = p.idx[(size_t)t * p.k + s];
        const bool e_ok = e >= 0 && e < p.E;
        int row = -1;
        if (p.compute_rows) {
          if (e_ok) row = p.dst_row0[e] + p.blk_base[(size_t)(t / ROUTER_TOKENS) * p.E + e] + p.within[(size_t)t * p.k + s];
          if (lane == 0) p.rows[(size_t)t * p.k + s] = row;
        } else {
          row = p.rows[(size_t)t * p.k + s];
        }
        if (e_ok && row >= 0 && row < p.cap) drow[s] = reinterpret_cast<uint4*>(p.dst[e / p.LE] + (size_t)row * p.H);
        else if (lane == 0) { if (e_ok && row >= p.cap) moe_overflow((unsigned)row + 1u); else moe_fail(4u, (unsigned)row); }
        if (p.scale) sc[s] = p.scale[(size_t)t * p.k + s];
      }
    }
    for (int v = lane; v < nvec; v += 32) {
      const uint4 raw = sr[v];
      if (p.scale) {
        float f[8];
        unpack8(raw, f);
#pragma unroll
        for (int s = 0; s < MOE_MAX_TOPK; s++) {
          if (s < p.k && drow[s]) {
            float g[8];
#pragma unroll
            for (int i = 0; i < 8; i++) g[i] = f[i] * sc[s];
            drow[s][v] = pack8(g);
          }
        }
      } else {
#pragma unroll
        for (int s = 0; s < MOE_MAX_TOPK; s++)
          if (s < p.k && drow[s]) drow[s][v] = raw;
      }
    }
  }
  // every store of this CTA is fenced, then the CTA counts itself at every destination
  __threadfence_system();
  __syncthreads();
  if (threadIdx.x < p.n) {
    __threadfence_system();
    lbcomm::red_release_sys_add(p.arrive[threadIdx.x], 1u);
  }
}

// -------------------------------------------------------------------------------------------
// Pull: out[t] = sum_s w[t, s] * src_owner[row(t, s)];  dots[t, s] = <src_owner[row(t, s)], dots_with[t]>
// -------------------------------------------------------------------------------------------
struct PullParams {
  bf16* out;                // [T, H] or null
  const bf16* add;          // [T, H] or null: added to out
  const float* w;           // [T, k] or null (weights 1)
  const int* idx;           // [T, k]
  const int* rows;          // [T, k]
  float* dots;              // [T, k] or null
  const bf16* dots_with;    // [T, H] (with dots)
  const bf16* src[MOE_MAX_RANKS];
  unsigned int* ready[MOE_MAX_RANKS];    // rank r's "source buffer of rank q is complete" words [n]
  unsigned int epoch;
  unsigned long long wait_ns;
  int T, H, E, LE, k, n, me, cap;
};

// Bound by the latency of its loads: a token is one warp's.  KS is the smallest of 1, 2, 4, 8 that holds k; a warp has eight row vectors in
// flight, 8 / KS from each of its rows, before it adds the first.  (With a branch per slot and vector, every load was waited for by
// itself: T 4096, H 2048, k 2 31 us, now 16.)  A sum takes its terms in the same order for every KS.
template <int KS>
__global__ void __launch_bounds__(256) moe_pull_kernel(const PullParams p) {
  if (p.n == 1) grid_go();
  grid_wait();
  constexpr int U = 8 / KS;
  __shared__ int s_fail;
  if (threadIdx.x == 0) s_fail = 0;
  __syncthreads();
  // this kernel runs behind the kernel that produced this rank's source buffer: tell every peer,
  // then wait until every peer's buffer is complete too
  if (threadIdx.x < p.n) {
    if (blockIdx.x == 0) {
      __threadfence_system();
      lbcomm::st_release_sys(p.ready[threadIdx.x] + p.me, p.epoch);
    }
    if (!lbcomm::flag_wait_ge(p.ready[p.me] + threadIdx.x, p.epoch, p.wait_ns)) { s_fail = 1; moe_fail(2u, 2u); }
  }
  __syncthreads();
  if (s_fail) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
  const int nvec = p.H >> 3;
  for (int t = blockIdx.x * wpb + warp; t < p.T; t += gridDim.x * wpb) {
    const uint4* srow[KS];
    float wt[KS], dot[KS];
#pragma unroll
    for (int s = 0; s < KS; s++) {
      srow[s] = nullptr;
      wt[s] = 1.f;
      dot[s] = 0.f;
      if (s < p.k) {
        const int e = p.idx[(size_t)t * p.k + s];
        const int row = p.rows[(size_t)t * p.k + s];
        if (e >= 0 && e < p.E && row >= 0 && row < p.cap)
          srow[s] = reinterpret_cast<const uint4*>(p.src[e / p.LE] + (size_t)row * p.H);
        else if (lane == 0 && !(e >= 0 && e < p.E && row >= p.cap)) moe_fail(5u, (unsigned)row);   // beyond capacity: dropped at dispatch
        if (p.w) wt[s] = p.w[(size_t)t * p.k + s];
      }
    }
    const uint4* dw = p.dots ? reinterpret_cast<const uint4*>(p.dots_with + (size_t)t * p.H) : nullptr;
    uint4* orow = p.out ? reinterpret_cast<uint4*>(p.out + (size_t)t * p.H) : nullptr;
    const uint4* arow = p.add ? reinterpret_cast<const uint4*>(p.add + (size_t)t * p.H) : nullptr;
    for (int v0 = lane; v0 < nvec; v0 += 32 * U) {
      uint4 raw[U][KS], with[U];                                      // `with`: the row of dots_with or of `add` (never both)
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int v = v0 + 32 * u;
        if (v >= nvec) continue;
        if (dw) with[u] = dw[v];
        else if (arow) with[u] = arow[v];
#pragma unroll
        for (int s = 0; s < KS; s++)
          if (srow[s]) raw[u][s] = lbcomm::ld_nc_v4(srow[s] + v);
      }
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int v = v0 + 32 * u;
        if (v >= nvec) continue;
        float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        float g[8];
        if (dw || arow) unpack8(with[u], g);
#pragma unroll
        for (int s = 0; s < KS; s++) {
          if (srow[s]) {
            float f[8];
            unpack8(raw[u][s], f);
#pragma unroll
            for (int i = 0; i < 8; i++) acc[i] = fmaf(wt[s], f[i], acc[i]);
            if (dw) {
#pragma unroll
              for (int i = 0; i < 8; i++) dot[s] = fmaf(f[i], g[i], dot[s]);
            }
          }
        }
        if (arow) {
#pragma unroll
          for (int i = 0; i < 8; i++) acc[i] += g[i];
        }
        if (orow) orow[v] = pack8(acc);
      }
    }
    if (p.dots) {
#pragma unroll
      for (int s = 0; s < KS; s++) {
        if (s < p.k) {
          const float d = warp_sum(dot[s]);
          if (lane == 0) p.dots[(size_t)t * p.k + s] = d;
        }
      }
    }
  }
}

// -------------------------------------------------------------------------------------------
// Router backward
// -------------------------------------------------------------------------------------------
// A block takes 64 tokens x 256 columns: warp w the tokens 8 w .. 8 w + 7, a lane 8 columns.  A warp's tokens stay in registers over
// the experts, whose gate weights are fetched once for all of them, and the block's share of the gate gradient is summed over its
// warps in shared memory before one vector reduction per 4 columns (four atomics where the gradient does not start on 16 bytes).
// (A block per 64 tokens and all columns left most SMs idle and fetched the weights again for every token: T 4096, H 2048, inputs
// not in L2, E 8 108 us, now 35; E 64 688, now 184.)
constexpr int RB_TOKENS = 64, RB_COLS = 256, RB_WARPS = 8, RB_TPW = RB_TOKENS / RB_WARPS;

__global__ void __launch_bounds__(RB_WARPS * 32)
moe_router_bwd_kernel(const bf16* __restrict__ x, const bf16* __restrict__ wg, const float* __restrict__ probs,
                      const int* __restrict__ idx, const float* __restrict__ dwts, const float* __restrict__ frac,
                      const float* __restrict__ daux, bf16* __restrict__ dx, float* __restrict__ dwg_acc, int T, int H,
                      int E, int k) {
  grid_go();
  grid_wait();
  __shared__ float s_dl[RB_TOKENS][MOE_MAX_EXPERTS + 1];
  __shared__ __align__(16) float s_w[RB_WARPS][RB_COLS];
  const int t0 = blockIdx.x * RB_TOKENS;
  const int ntok = min(RB_TOKENS, T - t0);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const float aux_c = daux ? daux[0] * (float)E / (float)T : 0.f;
  // dlogit[t, e] = p (dp - sum_e' p dp) with dp = routed-weight gradient + load-balance term
  for (int i = threadIdx.x; i < RB_TOKENS; i += blockDim.x) {
    const int t = t0 + i;
    if (i >= ntok) {
      for (int e = 0; e < E; e++) s_dl[i][e] = 0.f;
      continue;
    }
    int ch[MOE_MAX_TOPK];
    float cw[MOE_MAX_TOPK];
#pragma unroll
    for (int s = 0; s < MOE_MAX_TOPK; s++) {
      ch[s] = s < k ? idx[(size_t)t * k + s] : -1;
      cw[s] = s < k ? dwts[(size_t)t * k + s] : 0.f;
    }
    float dot = 0.f;
    for (int e = 0; e < E; e++) {
      float dp = aux_c * frac[e];
#pragma unroll
      for (int s = 0; s < MOE_MAX_TOPK; s++) if (ch[s] == e) dp += cw[s];
      s_dl[i][e] = dp;
      dot += probs[(size_t)t * E + e] * dp;
    }
    for (int e = 0; e < E; e++) s_dl[i][e] = probs[(size_t)t * E + e] * (s_dl[i][e] - dot);
  }
  __syncthreads();
  const int nvec = H >> 3, v = blockIdx.y * 32 + lane;
  const bool in = v < nvec;
  uint4 xr[RB_TPW];
  float dxa[RB_TPW][8];
#pragma unroll
  for (int i = 0; i < RB_TPW; i++) {
    const int tl = warp * RB_TPW + i;
    xr[i] = in && tl < ntok ? reinterpret_cast<const uint4*>(x + (size_t)(t0 + tl) * H)[v] : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int j = 0; j < 8; j++) dxa[i][j] = 0.f;
  }
  for (int e = 0; e < E; e++) {
    const uint4 wr = in ? __ldg(reinterpret_cast<const uint4*>(wg + (size_t)e * H) + v) : make_uint4(0, 0, 0, 0);
    float wf[8], acc[8];
    unpack8(wr, wf);
#pragma unroll
    for (int j = 0; j < 8; j++) acc[j] = 0.f;
#pragma unroll
    for (int i = 0; i < RB_TPW; i++) {
      const float d = s_dl[warp * RB_TPW + i][e];
      float xf[8];
      unpack8(xr[i], xf);
#pragma unroll
      for (int j = 0; j < 8; j++) {
        dxa[i][j] = fmaf(d, wf[j], dxa[i][j]);       // dx[t, cols] = sum_e dlogit[t, e] wg[e, cols]
        acc[j] = fmaf(d, xf[j], acc[j]);             // dwg[e, cols] += sum_t dlogit[t, e] x[t, cols]
      }
    }
    __syncthreads();                                 // the previous expert's sums have been read
    *reinterpret_cast<float4*>(&s_w[warp][lane * 8]) = make_float4(acc[0], acc[1], acc[2], acc[3]);
    *reinterpret_cast<float4*>(&s_w[warp][lane * 8 + 4]) = make_float4(acc[4], acc[5], acc[6], acc[7]);
    __syncthreads();
    if (threadIdx.x < RB_COLS / 4 && blockIdx.y * RB_COLS + threadIdx.x * 4 < H) {
      float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int w = 0; w < RB_WARPS; w++) {
        const float4 a = *reinterpret_cast<const float4*>(&s_w[w][threadIdx.x * 4]);
        sum.x += a.x; sum.y += a.y; sum.z += a.z; sum.w += a.w;
      }
      float* dst = dwg_acc + (size_t)e * H + blockIdx.y * RB_COLS + threadIdx.x * 4;
      if (((uintptr_t)dwg_acc & 15) == 0) {
        asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(sum.x), "f"(sum.y), "f"(sum.z), "f"(sum.w)
                     : "memory");
      } else {
        atomicAdd(dst, sum.x); atomicAdd(dst + 1, sum.y); atomicAdd(dst + 2, sum.z); atomicAdd(dst + 3, sum.w);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < RB_TPW; i++) {
    const int tl = warp * RB_TPW + i;
    if (in && tl < ntok) reinterpret_cast<uint4*>(dx + (size_t)(t0 + tl) * H)[v] = pack8(dxa[i]);
  }
}

int moe_grid(int T) {
  int blocks = (T + 7) / 8;
  const int cap = lb_num_sms() * 4;
  if (blocks > cap) blocks = cap;
  return blocks < 1 ? 1 : blocks;
}

}  // namespace

extern "C" int lb_moe_status(void* out) {
  cudaError_t e = cudaMemcpyFromSymbol(out, g_moe_status, sizeof(unsigned int) * 4);
  if (e != cudaSuccess) { g_lb_last_cuda_error = (int)e; return LB_ERR_LAUNCH; }
  unsigned int zeros[4] = {0, 0, 0, 0};
  cudaMemcpyToSymbol(g_moe_status, zeros, sizeof(zeros));
  return LB_OK;
}

// Number of router blocks (rows of blk_hist / blk_psum / blk_base) for T tokens.
extern "C" int lb_moe_router_blocks(int T) { return (T + ROUTER_TOKENS - 1) / ROUTER_TOKENS; }

// Number of CTAs lb_moe_push launches for T tokens on this device: every destination's arrival word
// grows by this much per source rank and call.
extern "C" int lb_moe_push_ctas(int T) { return moe_grid(T); }

// x [T, H] bf16, wg [E, H] bf16 -> probs [T, E] fp32, idx [T, k] int32, wts [T, k] fp32 (softmax
// probabilities of the chosen experts), within [T, k] int32, blk_hist [nblk, E] int32,
// blk_psum [nblk, E] fp32.  E <= 64, k <= 8, H a multiple of 8.
extern "C" int lb_moe_router(const void* x, const void* wg, int T, int H, int E, int k, void* probs, void* idx, void* wts,
                             void* within, void* blk_hist, void* blk_psum, void* stream) {
  if (T <= 0 || (H % 8) || E < 1 || E > MOE_MAX_EXPERTS || k < 1 || k > MOE_MAX_TOPK || k > E) return LB_ERR_SHAPE;
  // One token at a time where a warp has no second one, four elsewhere.  One / four, us, single launches between events with inputs that
  // are not in L2: T 1, H 2048, E 8 16 / 19; T 16384, H 4096, E 64 766 / 402; T 32768, H 2048, E 64 625 / 369.  (The form that waited for each load by
  // itself took 25, 808 and 664 under the same conditions; with inputs in L2 T 1 takes 17, it took 19.)
  const bool one = T <= ROUTER_THREADS / 32;
  LB_LAUNCH(one ? moe_router_kernel<1> : moe_router_kernel<4>, lb_moe_router_blocks(T), ROUTER_THREADS, 0, (cudaStream_t)stream, (const bf16*)x,
            (const bf16*)wg, T, H, E, k, (float*)probs, (int*)idx, (float*)wts, (int*)within, (int*)blk_hist, (float*)blk_psum);
  return LB_OK;
}

// cnt_ptrs[r] / flag_ptrs[r]: rank r's count table [2][n][E] int32 and "counts arrived" words [n]
// (peer-visible, zeroed once); epoch grows by one per call, parity alternates.  seg has 2 * LE + 2
// ints: segment offsets, segment counts, padded end of the last segment, rows received.
extern "C" int lb_moe_plan(const void* blk_hist, const void* blk_psum, void* blk_base, void* dst_row0, void* seg,
                           void* frac, void* aux, int nblk, int E, int n, int me, int T, int k, int cap,
                           void* const* cnt_ptrs, void* const* flag_ptrs, int parity, unsigned int epoch, void* stream) {
  if (n < 1 || n > MOE_MAX_RANKS || E < 1 || E > MOE_MAX_EXPERTS || (E % n) || me < 0 || me >= n) return LB_ERR_SHAPE;
  PlanParams p;
  p.blk_hist = (const int*)blk_hist; p.blk_psum = (const float*)blk_psum; p.blk_base = (int*)blk_base;
  p.dst_row0 = (int*)dst_row0; p.seg = (int*)seg; p.frac = (float*)frac; p.aux = (float*)aux;
  p.nblk = nblk; p.E = E; p.LE = E / n; p.n = n; p.me = me; p.T = T; p.k = k; p.cap = cap;
  for (int r = 0; r < n; r++) { p.cnt_all[r] = (int*)cnt_ptrs[r]; p.flags[r] = (unsigned int*)flag_ptrs[r]; }
  p.parity = parity & 1; p.epoch = epoch; p.wait_ns = g_lb_flag_wait_ns;
  return lb_launch_cluster(n == 1, 1, moe_plan_kernel, 1, 256, 0, (cudaStream_t)stream, p);
}

// dst_ptrs[r] / arrive_ptrs[r]: rank r's destination buffer [cap, H] bf16 and its arrival word.
// compute_rows != 0: rows[t, s] is computed from (within, blk_base, dst_row0) and written;
// otherwise rows is read.  scale [T, k] fp32 or null.  Launches lb_moe_push_ctas(T) CTAs.
extern "C" int lb_moe_push(const void* src, const void* scale, const void* idx, const void* within, const void* blk_base,
                           const void* dst_row0, void* rows, const void* seg, int T, int H, int E, int k, int n, int me,
                           int cap, int compute_rows, void* const* dst_ptrs, void* const* arrive_ptrs, void* stream) {
  if (T <= 0 || (H % 8) || n < 1 || n > MOE_MAX_RANKS || E < 1 || E > MOE_MAX_EXPERTS || (E % n) || k < 1 || k > MOE_MAX_TOPK)
    return LB_ERR_SHAPE;
  PushParams p;
  p.src = (const bf16*)src; p.scale = (const float*)scale; p.idx = (const int*)idx; p.within = (const int*)within;
  p.blk_base = (const int*)blk_base; p.dst_row0 = (const int*)dst_row0; p.rows = (int*)rows; p.seg = (const int*)seg;
  for (int r = 0; r < n; r++) { p.dst[r] = (bf16*)dst_ptrs[r]; p.arrive[r] = (unsigned int*)arrive_ptrs[r]; }
  p.own = p.dst[me];
  p.T = T; p.H = H; p.E = E; p.LE = E / n; p.k = k; p.n = n; p.me = me; p.cap = cap; p.compute_rows = compute_rows;
  return lb_launch_cluster(n == 1, 1, moe_push_kernel, moe_grid(T), 256, 0, (cudaStream_t)stream, p);
}

// src_ptrs[r]: rank r's source buffer [cap, H] bf16; ready_ptrs[r]: rank r's ready words [n] for
// this buffer; epoch grows by one per call on this buffer.  out [T, H] or null; w [T, k] or null;
// dots [T, k] with dots_with [T, H], or both null.  add [T, H] or null (not together with dots): out is the sum plus `add`, rounded once.
extern "C" int lb_moe_pull_add(void* out, const void* add, const void* w, const void* idx, const void* rows, void* dots, const void* dots_with,
                               int T, int H, int E, int k, int n, int me, int cap, void* const* src_ptrs,
                               void* const* ready_ptrs, unsigned int epoch, void* stream) {
  if (T <= 0 || (H % 8) || n < 1 || n > MOE_MAX_RANKS || E < 1 || E > MOE_MAX_EXPERTS || (E % n) || k < 1 || k > MOE_MAX_TOPK)
    return LB_ERR_SHAPE;
  if ((dots == nullptr) != (dots_with == nullptr) || (add && (dots || !out))) return LB_ERR_ARG;
  PullParams p;
  p.out = (bf16*)out; p.add = (const bf16*)add; p.w = (const float*)w; p.idx = (const int*)idx; p.rows = (const int*)rows; p.dots = (float*)dots;
  p.dots_with = (const bf16*)dots_with;
  for (int r = 0; r < n; r++) { p.src[r] = (const bf16*)src_ptrs[r]; p.ready[r] = (unsigned int*)ready_ptrs[r]; }
  p.epoch = epoch; p.wait_ns = g_lb_flag_wait_ns;
  p.T = T; p.H = H; p.E = E; p.LE = E / n; p.k = k; p.n = n; p.me = me; p.cap = cap;
  return lb_launch_cluster(n == 1, 1, k == 1 ? moe_pull_kernel<1> : k == 2 ? moe_pull_kernel<2> : k <= 4 ? moe_pull_kernel<4> : moe_pull_kernel<8>,
                           moe_grid(T), 256, 0, (cudaStream_t)stream, p);
}

extern "C" int lb_moe_pull(void* out, const void* w, const void* idx, const void* rows, void* dots, const void* dots_with,
                           int T, int H, int E, int k, int n, int me, int cap, void* const* src_ptrs,
                           void* const* ready_ptrs, unsigned int epoch, void* stream) {
  return lb_moe_pull_add(out, nullptr, w, idx, rows, dots, dots_with, T, H, E, k, n, me, cap, src_ptrs, ready_ptrs, epoch, stream);
}

// dwts [T, k] fp32: gradient of the loss with respect to the routed weights; daux: device pointer to
// the gradient with respect to the load-balance loss (or null); frac [E] from lb_moe_plan.
// dx [T, H] bf16 is written; dwg_acc [E, H] fp32 is added to (zero it first).
extern "C" int lb_moe_router_bwd(const void* x, const void* wg, const void* probs, const void* idx, const void* dwts,
                                 const void* frac, const void* daux, void* dx, void* dwg_acc, int T, int H, int E, int k,
                                 void* stream) {
  if (T <= 0 || (H % 8) || E < 1 || E > MOE_MAX_EXPERTS || k < 1 || k > MOE_MAX_TOPK) return LB_ERR_SHAPE;
  const dim3 grid((T + RB_TOKENS - 1) / RB_TOKENS, (H + RB_COLS - 1) / RB_COLS);
  LB_LAUNCH(moe_router_bwd_kernel, grid, RB_WARPS * 32, 0, (cudaStream_t)stream, (const bf16*)x, (const bf16*)wg, (const float*)probs,
            (const int*)idx, (const float*)dwts, (const float*)frac, (const float*)daux, (bf16*)dx, (float*)dwg_acc, T, H, E, k);
  return LB_OK;
}
