// bf16 GEMM for launches that do not fill the chip:  C[M,N] (+)= op(A) op(B)^T with tiles of 128 x 64 whose reduction may be
// split over a cluster of 2, 4 or 8 CTAs; one or two problems per launch.
//
// Why: with the 128 x 256 tiles of gemm_grouped.cu a small problem is a handful of CTAs, each of which streams its whole K through
// one SM.  An SM brings in 130 to 150 GB/s (what it has in flight over the latency of memory), so 0.38 us per 64 of K is all that such a launch
// takes, whatever its other sizes.  Smaller tiles and a split K spread the same bytes over the chip, tiles are named by blockIdx (no
// list to fetch first), and two CTAs share an SM.  Rows x columns x depth, operands from memory, 128x256 tiles / this, us: 128 x 2304 x 768
// 11.7 / 8.0, 128 x 768 x 2048 17.2 / 7.4, 128 x 2048 x 5632 32.7 / 12.8, 1000 x 768 x 2048 18.3 / 12.4; data and weight gradient of
// 1000 x 768 x 768 13.2 / 10.1.  What is left (6 us for the shortest): launch, barriers and tensor memory, one round trip to memory, stores.
//
// A CTA of a split tile leaves the sum over its part of K in tensor memory.  It sends the columns that another CTA of the cluster owns into that one's
// shared memory, where they are counted on a barrier, and adds what it receives to its own in the order of the parts: the result does not depend on
// timing.  Roles, pipeline, descriptors and epilogues are those of gemm_grouped.cu.  Cycles from the end of the wait for the kernel before (clock64, 128 x
// 768 x 768 in 4 parts): first stage 1800, accumulator 3050; then 5300 for two cluster barriers, eight columns at a time and a loop over the parts,
// which is why the parts are a template's, the columns come in one load and the sums are counted on a barrier.  128 x 2304 x 768 with the rotation: 7300
// of 13900 cycles were its tables, fetched per eight columns; they are now on their way while the MMAs run.
// A launch starts under the kernel before it (grid_go(), grid_wait()), and asks for its part of B, which that kernel hardly ever writes, to be brought to
// L2 meanwhile: the 99 kernels of 12 layers of 768 columns over 128 tokens 575 us launched one after the other, 521 so, 495 with the request.  (The 87 kernels of the same without gradients: 486, and 471 with what the paragraph above changed.)
// Every wait is bounded; on expiry the kernel records a status code (lb_gemm_split_status), stops issuing work, frees its TMEM and returns.
#include <algorithm>
#include "gemm_split.h"
#include "tcgen05.cuh"

static __device__ unsigned int g_split_status[4] = {0, 0, 0, 0};

namespace {

constexpr int BM = 128, BN = 64, BK = 64;
constexpr int HB = BN / 2;                               // columns of a tile's two blocks
constexpr int A_BYTES = BM * BK * 2, B_BYTES = BN * BK * 2;
constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
// KS parts of K.  A tile's 8 groups of 8 columns are finished by its CTAs: NG groups of each block by everyone, or, with eight parts, one group each (no
// activation then, which wants both blocks' columns in one CTA).  With four and more a CTA has few k-blocks at a time in flight, and the place of a
// fourth stage is where the others' sums arrive.
template <int KS>
struct Cfg {
  static constexpr int STAGES = KS >= 4 ? 3 : 4;
  static constexpr int G = 8 / KS, NG = KS == 8 ? 1 : HB / 8 / KS, NB = G / NG;      // groups of a CTA: NB blocks, NG in each
  // Groups of a block that a warp finishes.  Where a CTA has one of each block, one warp takes the first block's and one the second's; the pair (activation), or
  // the only one, is the first warp's.
  static constexpr int GW = NG > 1 ? NG / 2 : 1;
  static constexpr int RECV_BYTES = (KS - 1) * BM * G * 8 * 4;
  static constexpr int OFF_RECV = STAGES * STAGE_BYTES;
  static constexpr int OFF_BAR = OFF_RECV + RECV_BYTES;
  static constexpr int SMEM_BYTES = OFF_BAR + 256;
  static_assert(2 * (SMEM_BYTES + 1024) <= 233472, "two CTAs per SM");
};
// Warps 0 and 1 load and multiply, the others finish, two for each 32 rows: a warp's epilogue is one chain of instructions, not a stream that the SM's units
// bound, so half of the columns take half of the time (one / two warps for 32 rows, forward
// and backward, us: MLP of 16 x 768 46.2 / 42.1, 64 x 1024 60.5 / 59.5, 100 x 768 48.4 / 47.1, attention layer of 512 x 768 57.2 / 54.7; 12 layers of 128 x 768
// forward 461.7 / 454.5; equal where the tiles are many).
constexpr int NUM_THREADS = 320;
constexpr int MAX_PROBLEMS = 2;
constexpr int PREFETCH = 16;                             // k-blocks of B that a CTA asks for ahead of its start (38 MB of all CTAs that run at a time)

// epi: 0 C = acc (+ C); 1 gate | up -> C (not stored where C is null), silu(g) * u -> C2; 2 dh -> dg | du with g | u from C2; 4 rotation (as in
// gemm_grouped.cu).
struct Problem {
  bf16* C;
  long long ldc;
  bf16* C2;
  long long ldc2;
  int M, N, a_mn, b_mn, accumulate, epi, half;
  int tiles_m, num_kb, first;                            // `first`: tiles of the problems before this one
  int a_rows;                                            // rows of an A tile that are loaded: all 128, or those of a smaller matrix
};
struct Params {
  CUtensorMap ta[MAX_PROBLEMS], tb[MAX_PROBLEMS];
  Problem prob[MAX_PROBLEMS];
  RopeArgs rope;
  int np;
};

__device__ __forceinline__ void give_up(volatile int* abort_flag, unsigned where) {
  *abort_flag = 1;
  atomicExch(&g_split_status[0], 1u);
  atomicExch(&g_split_status[1], where);
}

template <int STAGES, bool A_MN, bool B_MN>
__device__ __forceinline__ bool produce(const CUtensorMap* ta, const CUtensorMap* tb, int m0, int n0, int n1, int a_rows, int kb0, int n_kb,
                                        uint32_t smem_base, uint32_t bar_base, volatile int* abort_flag) {
  int stage = 0;
  uint32_t phase = 0;
  for (int kb = kb0; kb < kb0 + n_kb; kb++) {
    if (!bw::mbar_wait(bar_base + 8u * (STAGES + stage), phase ^ 1u, abort_flag)) return false;
    const uint32_t fb = bar_base + 8u * stage;
    bw::mbar_expect_tx(fb, a_rows * BK * 2 + B_BYTES);
    const uint32_t sa = smem_base + stage * STAGE_BYTES, sb = sa + A_BYTES;
    const int k0 = kb * BK;
    if (!A_MN) {
      bw::tma_load_2d(sa, ta, k0, m0, fb);                                                      // box {64 k, a_rows m}
    } else {
      bw::tma_load_2d(sa, ta, m0, k0, fb);                                                      // boxes {64 m, 64 k}
      if (a_rows > 64) bw::tma_load_2d(sa + 8192, ta, m0 + 64, k0, fb);
    }
    if (!B_MN) {
      bw::tma_load_2d(sb, tb, k0, n0, fb);                                                      // boxes {64 k, 32 n}
      bw::tma_load_2d(sb + HB * BK * 2, tb, k0, n1, fb);
    } else {
      bw::tma_load_2d(sb, tb, n0, k0, fb);                                                      // box {64 n, 64 k}
    }
    if (++stage == STAGES) { stage = 0; phase ^= 1u; }
  }
  return true;
}

template <int STAGES, bool A_MN, bool B_MN>
__device__ __forceinline__ bool multiply(uint32_t d_tmem, int n_kb, uint32_t smem_base, uint32_t bar_base, volatile int* abort_flag) {
  constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((A_MN ? 1u : 0u) << 15) | ((B_MN ? 1u : 0u) << 16) |
                             ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
  constexpr uint32_t a_lbo = A_MN ? 8192u : 16u, b_lbo = B_MN ? 8192u : 16u;
  constexpr uint32_t a_kstep = A_MN ? 2048u : 32u, b_kstep = B_MN ? 2048u : 32u;   // bytes per K=16 slice
  int stage = 0;
  uint32_t phase = 0;
  for (int kb = 0; kb < n_kb; kb++) {
    if (!bw::mbar_wait(bar_base + 8u * stage, phase, abort_flag)) return false;
    bw::fence_after();
    const uint32_t sa = smem_base + stage * STAGE_BYTES, sb = sa + A_BYTES;
#pragma unroll
    for (int k = 0; k < BK / 16; k++)
      bw::umma_bf16(d_tmem, bw::make_desc(sa + k * a_kstep, a_lbo, 1024u), bw::make_desc(sb + k * b_kstep, b_lbo, 1024u), idesc,
                    (kb | k) ? 1u : 0u);
    bw::umma_commit(bar_base + 8u * (STAGES + stage));         // frees this smem stage when the MMAs have read it
    if (++stage == STAGES) { stage = 0; phase ^= 1u; }
  }
  return true;
}

template <int KS>
__global__ void __launch_bounds__(NUM_THREADS, 2) gemm_split_kernel(const __grid_constant__ Params gp) {
  using C = Cfg<KS>;
  constexpr int STAGES = C::STAGES, NG = C::NG, NB = C::NB, GW = C::GW;
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t smem_base = bw::smem_u32(smem);
  const uint32_t bar_base = smem_base + C::OFF_BAR;
  const uint32_t tfull = bar_base + 8u * 2 * STAGES, received = tfull + 8;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + C::OFF_BAR + 8 * (2 * STAGES + 2));
  int* s_abort = reinterpret_cast<int*>(tmem_slot + 1);        // {abort, extra wait in ms}: see bw::mbar_wait
  volatile int* abort_flag = s_abort;
  int* s_sums = s_abort + 2;                                   // the same for the wait for the other parts' sums, which no abort cuts short
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0);      // (uniform over the warp)
  const int lane = threadIdx.x & 31;
  const int rank = KS > 1 ? (int)bw::cluster_ctarank() : 0;
  const int t = (int)blockIdx.x / KS;
  const int pi = gp.np > 1 && t >= gp.prob[1].first ? 1 : 0;
  const Problem& pr = gp.prob[pi];
  const int tl = t - pr.first;
  // rows fastest: the tiles that run together share their part of B, which is the weight more often than not
  const int m0 = (tl % pr.tiles_m) * BM, tn = tl / pr.tiles_m;
  // the tile's two blocks of columns: neighbours, or the gate and the up columns of the same index
  const int n0 = pr.epi == 1 ? tn * HB : tn * BN;
  const int n1 = pr.epi == 1 ? pr.half + n0 : n0 + HB;
  // group g of this warp in block b: which block, its place among the CTA's groups of a block, its first column, and whether the warp has that block
  const int set = warp >= 6 ? 1 : 0;
  auto block_of = [&](int b) { return KS == 8 ? rank >> 2 : b; };
  auto place_of = [&](int g) { return NG > 1 ? set * GW + g : g; };
  auto column_of = [&](int g) { return KS == 8 ? (rank & 3) * 8 : (rank * NG + place_of(g)) * 8; };
  auto mine = [&](int b) { return NG > 1 || (NB == 1 || pr.epi == 1 ? set == 0 : set == b); };
  const int kb0 = (int)((long long)pr.num_kb * rank / KS), n_kb = (int)((long long)pr.num_kb * (rank + 1) / KS) - kb0;

  if (threadIdx.x == 64) { bw::prefetch_tmap(&gp.ta[pi]); bw::prefetch_tmap(&gp.tb[pi]); }
  if (threadIdx.x == 0) {
    s_abort[0] = 0;
    s_abort[1] = 0;
    s_sums[0] = 0;
    s_sums[1] = 2000;                                          // (longer than another CTA's wait for its accumulator)
    if (smem_base & 1023u) { s_abort[0] = 1; atomicExch(&g_split_status[0], 4u); }      // the swizzled tiles need it: nothing is started
    for (int s = 0; s < STAGES; s++) {
      bw::mbar_init(bar_base + 8u * s, 1);
      bw::mbar_init(bar_base + 8u * (STAGES + s), 1);
    }
    bw::mbar_init(tfull, 1);
    bw::mbar_init(received, 1);
    bw::mbar_init_fence();
    if (KS > 1) bw::mbar_expect_tx(received, C::RECV_BYTES);
  }
  if (warp == 1) bw::tmem_alloc(bw::smem_u32(tmem_slot), BN);
  bw::fence_before();
  __syncthreads();
  if constexpr (KS > 1) bw::cluster_sync();                    // the peers' barriers exist before anything is sent
  bw::fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  bool ok = *abort_flag == 0;
  grid_go();
  if (warp == 2 && tl % pr.tiles_m == 0 && bw::elect_one()) {
    // B is the weight more often than not, and comes from memory: on its way to L2 while the kernel before this one still runs
    const CUtensorMap* tb = &gp.tb[pi];
    for (int kb = kb0; kb < kb0 + min(n_kb, PREFETCH); kb++) {
      if (pr.b_mn) {
        bw::tma_prefetch_2d(tb, n0, kb * BK);
      } else {
        bw::tma_prefetch_2d(tb, kb * BK, n0);
        bw::tma_prefetch_2d(tb, kb * BK, n1);
      }
    }
  }
  grid_wait();

  const int quad = warp & 3, row_in = quad * 32 + lane;
  const int row = m0 + row_in;
  const bool row_ok = row < pr.M;
  const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16);
  float rot[NB][GW][8];                                        // epi 4: cosines and sines of this row's columns, loaded ahead
  if (warp == 0) {
    if (ok && bw::elect_one()) {
      const CUtensorMap *ta = &gp.ta[pi], *tb = &gp.tb[pi];
      switch (pr.a_mn * 2 + pr.b_mn) {
        case 0: ok = produce<STAGES, false, false>(ta, tb, m0, n0, n1, pr.a_rows, kb0, n_kb, smem_base, bar_base, abort_flag); break;
        case 1: ok = produce<STAGES, false, true>(ta, tb, m0, n0, n1, pr.a_rows, kb0, n_kb, smem_base, bar_base, abort_flag); break;
        case 2: ok = produce<STAGES, true, false>(ta, tb, m0, n0, n1, pr.a_rows, kb0, n_kb, smem_base, bar_base, abort_flag); break;
        default: ok = produce<STAGES, true, true>(ta, tb, m0, n0, n1, pr.a_rows, kb0, n_kb, smem_base, bar_base, abort_flag); break;
      }
      if (!ok) give_up(abort_flag, 1u);
    }
  } else if (warp == 1) {
    if (ok && bw::elect_one()) {
      switch (pr.a_mn * 2 + pr.b_mn) {
        case 0: ok = multiply<STAGES, false, false>(tmem_base, n_kb, smem_base, bar_base, abort_flag); break;
        case 1: ok = multiply<STAGES, false, true>(tmem_base, n_kb, smem_base, bar_base, abort_flag); break;
        case 2: ok = multiply<STAGES, true, false>(tmem_base, n_kb, smem_base, bar_base, abort_flag); break;
        default: ok = multiply<STAGES, true, true>(tmem_base, n_kb, smem_base, bar_base, abort_flag); break;
      }
      if (ok) bw::umma_commit(tfull);                          // accumulator complete
      else give_up(abort_flag, 2u);
    }
  } else {
    if (pr.epi == 4) {
      const int pos = row_ok ? rope_position(gp.rope, row) : 0;
#pragma unroll
      for (int b = 0; b < NB; b++)
#pragma unroll
        for (int g = 0; g < GW; g++) {
          const int col = (block_of(b) ? n1 : n0) + column_of(g);
          if (mine(b) && col < gp.rope.cols) rope_load8(gp.rope, pos, col, rot[b][g]);
        }
    }
    if (ok && !bw::mbar_wait(tfull, 0, abort_flag)) { ok = false; give_up(abort_flag, 3u); }
    ok = __all_sync(0xffffffffu, ok);
  }
  __syncwarp();
  bw::fence_after();

  if constexpr (KS > 1) {
    if (warp >= 2) {
      // 8 columns at a time to the CTA that finishes them: a block of a quad's rows from either of its warps.  Every CTA sends all of its parts, zeros where
      // its accumulator did not come (the status word says that the result is void), and waits for all that is sent to it: a CTA that left out either could end,
      // or keep another from ending, while stores to its shared memory are on their way.
      const uint32_t here = smem_base + C::OFF_RECV + (uint32_t)(row_in * 16);
      uint32_t r[32];
      if (ok) {
        bw::tmem_ld32(taddr + set * HB, r);
        bw::tmem_ld_wait();
      } else {
#pragma unroll
        for (int i = 0; i < 32; i++) r[i] = 0;
      }
#pragma unroll
      for (int g = 0; g < 4; g++) {
        const int s = KS == 8 ? set * 4 + g : g / NG;          // the receiver; its place for this part: parts in order, its own left out
        if (s == rank) continue;
        const int slot = rank < s ? rank : rank - 1;
        const int to = KS == 8 ? 0 : set * NG + g % NG;
        const uint32_t dst = bw::cluster_addr(here + (uint32_t)((slot * C::G + to) * 8 * BM * 4), s);
        const uint32_t bar = bw::cluster_addr(received, s);
        bw::st_cluster_v4(dst, r + g * 8, bar);
        bw::st_cluster_v4(dst + BM * 16, r + g * 8 + 4, bar);
      }
    }
    __syncwarp();
    bw::cluster_arrive();
  }
  if (warp >= 2) {
    float f[NB][GW][8];
    if (ok) {
#pragma unroll
      for (int b = 0; b < NB; b++)
#pragma unroll
        for (int g = 0; g < GW; g++)
          if (mine(b)) bw::tmem_ld8(taddr + block_of(b) * HB + column_of(g), reinterpret_cast<uint32_t*>(f[b][g]));
      bw::tmem_ld_wait();
    }
    if constexpr (KS > 1) {
      // The sums order nothing but themselves: an acquire on their barrier, not a fence over the cluster beside it, and a barrier at the end that only keeps the CTA
      // there (12 layers of 128 x 768 471 -> 462 us, the MLP of 16 x 2048 81.5 -> 80.7; storing rows by neighbouring lanes gave 10 us of the first and 3 of the
      // second back, although the attention layer of 128 rows took 57.0 instead of 58.5).
      if (!bw::mbar_wait<true>(received, 0, s_sums)) { ok = false; give_up(abort_flag, 5u); }
      const float4* in = reinterpret_cast<const float4*>(smem + C::OFF_RECV) + row_in;
#pragma unroll
      for (int b = 0; b < NB; b++)
#pragma unroll
        for (int g = 0; g < GW; g++) {
          if (!mine(b)) continue;
          float own[8], sum[8];
#pragma unroll
          for (int i = 0; i < 8; i++) { own[i] = f[b][g][i]; sum[i] = 0.f; }
#pragma unroll
          for (int s = 0; s < KS; s++) {                       // in the order of the parts
            const int slot = s < rank ? s : s - 1;
            const float4* q = in + (size_t)((s == rank ? 0 : slot) * C::G + b * NG + place_of(g)) * 2 * BM;
            const float4 x = q[0], y = q[BM];
            const float part[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
#pragma unroll
            for (int i = 0; i < 8; i++) sum[i] += s == rank ? own[i] : part[i];
          }
#pragma unroll
          for (int i = 0; i < 8; i++) f[b][g][i] = sum[i];
        }
    }
    const int n_end = pr.epi == 1 ? pr.half : pr.N;
    if (row_ok && ok) {
#pragma unroll
      for (int g = 0; g < GW; g++) {
        const int cc = column_of(g);                           // column inside a block
        if (NB == 2 && pr.epi == 1) {
          // silu(g) * u is computed from the ROUNDED values (what a separate pass over the stored matrix would see)
          const int col = n0 + cc;
          if (mine(0) && col < n_end) {
            const uint4 pg = pack8(f[0][g]), pu = pack8(f[NB - 1][g]);
            if (pr.C) {
              bf16* grow = pr.C + (size_t)row * pr.ldc + col;
              *reinterpret_cast<uint4*>(grow) = pg;
              *reinterpret_cast<uint4*>(grow + pr.half) = pu;
            }
            float gt[8], u[8], h[8];
            unpack8(pg, gt);
            unpack8(pu, u);
#pragma unroll
            for (int i = 0; i < 8; i++) h[i] = gt[i] / (1.f + __expf(-gt[i])) * u[i];
            *reinterpret_cast<uint4*>(pr.C2 + (size_t)row * pr.ldc2 + col) = pack8(h);
          }
          continue;
        }
#pragma unroll
        for (int b = 0; b < NB; b++) {
          const int col = (block_of(b) ? n1 : n0) + cc;
          if (!mine(b) || col >= n_end) continue;
          bf16* dst = pr.C + (size_t)row * pr.ldc + col;
          if (pr.epi == 2) {
            const bf16* gu = pr.C2 + (size_t)row * pr.ldc2 + col;
            float d[8], gt[8], u[8], dg[8], du[8];
            unpack8(*reinterpret_cast<const uint4*>(gu), gt);
            unpack8(*reinterpret_cast<const uint4*>(gu + pr.half), u);
            unpack8(pack8(f[b][g]), d);                        // the value a stored bf16 dh would have had
#pragma unroll
            for (int i = 0; i < 8; i++) {
              const float sig = 1.f / (1.f + __expf(-gt[i]));
              dg[i] = d[i] * u[i] * sig * (1.f + gt[i] * (1.f - sig));
              du[i] = d[i] * gt[i] * sig;
            }
            *reinterpret_cast<uint4*>(dst) = pack8(dg);
            *reinterpret_cast<uint4*>(dst + pr.half) = pack8(du);
          } else {
            if (pr.accumulate) {
              float o[8];
              unpack8(*reinterpret_cast<const uint4*>(dst), o);
#pragma unroll
              for (int i = 0; i < 8; i++) f[b][g][i] += o[i];
            } else if (pr.epi == 4 && col < gp.rope.cols) {
              unpack8(pack8(f[b][g]), f[b][g]);                // the values a stored C would have
              rope_rotate8(rot[b][g], f[b][g]);
            }
            *reinterpret_cast<uint4*>(dst) = pack8(f[b][g]);
          }
        }
      }
    }
  }

  bw::fence_before();
  __syncthreads();
  if (warp == 1) {
    bw::fence_after();
    bw::tmem_dealloc(tmem_base, BN);
  }
  __syncwarp();
  if constexpr (KS > 1) bw::cluster_wait();                    // nobody has anything left to send to this CTA
}

template <int KS>
int launch(const Params& gp, long long tiles, cudaStream_t s) {
  static bool attr[64] = {false};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return LB_ERR_LAUNCH;
  if (!attr[dev]) {
    cudaFuncSetAttribute(gemm_split_kernel<KS>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<KS>::SMEM_BYTES);
    attr[dev] = true;
  }
  return lb_launch_cluster(true, KS, gemm_split_kernel<KS>, dim3((unsigned)(tiles * KS)), NUM_THREADS, Cfg<KS>::SMEM_BYTES, s, gp);
}

long long ceil_div(long long a, long long b) { return (a + b - 1) / b; }

}  // namespace

// Copies the status words of the split GEMM kernel to host memory and clears them.
extern "C" int lb_gemm_split_status(void* out) {
  cudaError_t e = cudaMemcpyFromSymbol(out, g_split_status, sizeof(unsigned int) * 4);
  if (e != cudaSuccess) { g_lb_last_cuda_error = (int)e; return LB_ERR_LAUNCH; }
  unsigned int zeros[4] = {0, 0, 0, 0};
  cudaMemcpyToSymbol(g_split_status, zeros, sizeof(zeros));
  return LB_OK;
}

// The arguments of lb_gemm_grouped_epi for n = 1 or 2 problems, with K split over ks = 1, 2, 4 or 8 CTAs (no more than a
// problem has 64-wide k-blocks; 8 without an activation).  lb_gemm_grouped_epi calls this with what gemm_split_parts() says.
extern "C" int lb_gemm_split(int n, const void* const* A, const void* const* B, void* const* C, const int* M, const int* N, const int* K,
                             const long long* lda, const long long* ldb, const long long* ldc, const int* a_mn, const int* b_mn,
                             const int* accumulate, const int* epi, void* const* C2, const long long* ldc2, const int* half, int ks, void* stream) {
  return gemm_split_rope(n, A, B, C, M, N, K, lda, ldb, ldc, a_mn, b_mn, accumulate, epi, C2, ldc2, half, ks, nullptr, stream);
}

int gemm_split_rope(int n, const void* const* A, const void* const* B, void* const* C, const int* M, const int* N, const int* K,
                    const long long* lda, const long long* ldb, const long long* ldc, const int* a_mn, const int* b_mn,
                    const int* accumulate, const int* epi, void* const* C2, const long long* ldc2, const int* half, int ks, const RopeArgs* rope,
                    void* stream) {
  if (n < 1 || n > MAX_PROBLEMS || (ks != 1 && ks != 2 && ks != 4 && ks != 8)) return LB_ERR_SHAPE;
  Params gp;
  gp.rope = rope ? *rope : RopeArgs{nullptr, nullptr, nullptr, 1, 64, 0};
  gp.np = n;
  long long tiles = 0;
  for (int i = 0; i < n; i++) {
    if (M[i] <= 0 || N[i] <= 0 || K[i] <= 0) return LB_ERR_SHAPE;
    if ((lda[i] % 8) || (ldb[i] % 8) || (ldc[i] % 8) || (N[i] % 8) || (a_mn[i] && (M[i] % 8))) return LB_ERR_SHAPE;
    if (((uintptr_t)A[i] | (uintptr_t)B[i] | (uintptr_t)C[i]) & 15) return LB_ERR_ARG;
    const int e = epi ? epi[i] : 0;
    if (e < 0 || e > 2 || (!C[i] && e != 1)) return LB_ERR_ARG;
    if (e) {
      if (!C2 || !ldc2 || !half || !C2[i] || ((uintptr_t)C2[i] & 15) || (ldc2[i] % 8) || half[i] <= 0 || (half[i] % 8)) return LB_ERR_ARG;
      if (e == 1 && (b_mn[i] || N[i] != 2 * half[i])) return LB_ERR_SHAPE;
      if (e == 2 && N[i] != half[i]) return LB_ERR_SHAPE;
      if (accumulate && accumulate[i]) return LB_ERR_ARG;
      if (ks == 8) return LB_ERR_SHAPE;
    }
    Problem& p = gp.prob[i];
    // the rows behind the last one of a short matrix are not loaded (what lies in the stage makes rows that are not stored): filling them
    // cost 16 x 11264 x 2048 27 instead of 15 us
    p.a_rows = M[i] >= BM ? BM : a_mn[i] ? (M[i] + 63) / 64 * 64 : (M[i] + 7) / 8 * 8;
    int rc;
    if (!a_mn[i]) rc = bw::make_map_bf16(&gp.ta[i], A[i], (uint64_t)K[i], (uint64_t)M[i], (uint64_t)lda[i], BK, (uint32_t)p.a_rows);
    else          rc = bw::make_map_bf16(&gp.ta[i], A[i], (uint64_t)M[i], (uint64_t)K[i], (uint64_t)lda[i], 64, BK);
    if (rc) return rc;
    if (!b_mn[i]) rc = bw::make_map_bf16(&gp.tb[i], B[i], (uint64_t)K[i], (uint64_t)N[i], (uint64_t)ldb[i], BK, HB);
    else          rc = bw::make_map_bf16(&gp.tb[i], B[i], (uint64_t)N[i], (uint64_t)K[i], (uint64_t)ldb[i], 64, BK);
    if (rc) return rc;
    p.C = (bf16*)C[i]; p.ldc = ldc[i]; p.C2 = e ? (bf16*)C2[i] : nullptr; p.ldc2 = e ? ldc2[i] : 0;
    p.M = M[i]; p.N = N[i]; p.a_mn = a_mn[i]; p.b_mn = b_mn[i]; p.accumulate = accumulate ? accumulate[i] : 0; p.epi = rope ? 4 : e; p.half = e ? half[i] : 0;
    p.tiles_m = (M[i] + BM - 1) / BM;
    p.num_kb = (K[i] + BK - 1) / BK;
    if (p.num_kb < ks) return LB_ERR_SHAPE;
    p.first = (int)tiles;
    tiles += p.tiles_m * (e == 1 ? ceil_div(half[i], HB) : ceil_div(N[i], BN));
    if (tiles * ks > (1 << 30)) return LB_ERR_SHAPE;
  }
  cudaStream_t s = (cudaStream_t)stream;
  switch (ks) {
    case 1: return launch<1>(gp, tiles, s);
    case 2: return launch<2>(gp, tiles, s);
    case 4: return launch<4>(gp, tiles, s);
    default: return launch<8>(gp, tiles, s);
  }
}

// Parts of K (1, 2, 4 or 8) with which this form is modelled to beat the list form of gemm_grouped.cu, or 0.  list_time: the latter's modelled
// time, in hundredths of a k-block.  Both models are in us and fitted to 189 launches in all forms (16 to 4096 rows, N 768 to 32000, K 16 to
// 5632; forward, data + weight gradient, activation epilogues; operands from memory): a fixed part, the k-blocks of a CTA, those that
// it waits for where there are more CTAs than SMs, the CTAs themselves, the bytes.  With the rule none of them is slower than the list form
// by more than it varies (2 %), they are 1.18x faster on average, and eleven stay up to 24 % behind the better form (the model sees
// 1000 x 2304 x 768 too late: 12.7, split 10.1).  Eight parts are for long reductions of few tiles (four / eight, us: 64 x 768 x 32000 46 / 28, 64 x 2048 x 11264
// 22 / 16, 64 x 1024 x 8192 16 / 10; where four already fill the chip, 64 x 4096 x 28672, 54 / 60), and not for activations.  `us` (or null) receives the
// modelled time of the form that is taken.
int gemm_split_parts(int n, const int* M, const int* N, const int* K, bool activation, int sms, long long list_time, double* us) {
  if (us) *us = 1e30;
  if (n < 1 || n > MAX_PROBLEMS || sms < 4) return 0;
  double mb = 0;
  long long min_kb = 1LL << 30;
  for (int i = 0; i < n; i++) {
    mb += 2e-6 * ((double)M[i] * K[i] + (double)N[i] * K[i] + (double)M[i] * N[i]);
    min_kb = std::min(min_kb, ceil_div(K[i], BK));
  }
  double best = 5.0 + 2.68e-3 * (double)list_time + 0.128 * mb;
  int parts = 0;
  for (int ks = 1; ks <= (activation || min_kb < 128 ? 4 : 8) && ks <= min_kb; ks *= 2) {
    double ctas = 0, work = 0, longest = 0;
    for (int i = 0; i < n; i++) {
      const double c = (double)ceil_div(M[i], BM) * ceil_div(N[i], BN) * ks, kb = (double)ceil_div(ceil_div(K[i], BK), ks);
      ctas += c;
      work += c * kb;
      longest = std::max(longest, kb);
    }
    const double t = 3.3 + 0.23 * longest + 0.113 * std::max(0.0, work / sms - longest) + 2.78 * ctas / sms + (ks > 1 ? 1.1 : 0.0) + 0.059 * mb;
    const double margin = ks == 8 ? 1.075 : 1.03;
    if (margin * t < best) { best = margin * t; parts = ks; }
  }
  if (us) *us = best;
  return parts;
}
