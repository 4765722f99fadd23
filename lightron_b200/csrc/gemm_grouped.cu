// Grouped bf16 GEMM for sm_100a: up to 8 independent problems  C_i[M_i,N_i] (+)= op(A_i) op(B_i)^T
// in ONE persistent launch.
//
// Why: a single GEMM whose tile count is not a multiple of the SM count leaves SMs idle in its
// last wave (a weight gradient [2560, 2048] has 160 tiles for 148 SMs: the second wave is 8 %
// full).  Launching the data gradient and the weight gradient of a linear layer together, or
// the GEMMs of all local experts of a MoE layer, gives the scheduler short tiles to fill those
// holes.  The host computes a static schedule (longest tiles first, each to the least loaded
// worker), uploads it once per shape, and every role of a worker walks the same list, so no
// intra-kernel tile broadcast is needed.  A worker is a CTA with tiles of 128x256 or a pair of CTAs
// (tcgen05 cta_group::2) with tiles of 256x256: Cfg has the two forms, choose_cg the choice.
//
// The main loop is the one of gemm_tcgen05.cu: TMA (128-byte swizzle, no multicast) -> mbarrier ring
// of 4 (CTA) or 5 to 6 (pair) stages -> tcgen05.mma 128x256x16 / 256x256x16 -> two 256-column TMEM accumulators
// per CTA -> tcgen05.ld epilogue overlapped with the next tile.  `accumulate` adds the old contents of C in
// the epilogue (gradient accumulation over micro-batches without a separate add).
// The ragged kernel (lb_gemm_ragged_epi, lb_gemm_ragged_wgrad) takes its tiles from device memory.
// Every wait is bounded; on expiry the kernel records a status code (lb_gemm_grouped_status),
// stops issuing work, frees its TMEM and returns.
#include <cuda.h>
#include <string.h>
#include <algorithm>
#include <cmath>
#include <map>
#include <mutex>
#include <queue>
#include <vector>
#include "common.cuh"
#include "tcgen05.cuh"
#include "comm.cuh"
#include "gemm_split.h"

static __device__ unsigned int g_grp_status[4] = {0, 0, 0, 0};

namespace {

constexpr int BM = 128, BN = 256, BK = 64;
constexpr int A_BYTES = BM * BK * 2;
constexpr int STG_BYTES = 32 * 128;      // 64 columns of the 32 rows of an epilogue warp
// CG CTAs work on one tile: 1 = a CTA per 128x256 tile, 2 = a pair (tcgen05 cta_group::2) per 256x256 tile, in which
// each CTA loads its 128 rows of A and half of B.  Per CTA a stage then holds 16 + 16 instead of 16 + 32 KB, and the tensor
// pipe, whose operand reads from shared memory are what limits and heats it, reads a third less.
// EW epilogue warps, each with a quarter of the accumulator's rows and all or half of its columns: four, or eight for launches with the SwiGLU
// backward, whose arithmetic is more than a warp per scheduler gets done in a main loop of K = 2048 (the others lose by eight: gate | up of 16384 x 2048 ->
// 5632 487 / 495 us, its gradients 1033 / 1060, those with the SwiGLU backward 606 / 545).
template <int CG, int EW>
struct Cfg {
  static constexpr int B_BYTES = BN / CG * BK * 2;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int STAGES = CG == 1 ? 4 : EW == 4 ? 6 : 5;
  static constexpr int NBUF = CG == 1 && EW == 8 ? 1 : 2;           // staging buffers of an epilogue warp
  static constexpr int OFF_STG = STAGES * STAGE_BYTES;
  static constexpr int OFF_BAR = OFF_STG + EW * NBUF * STG_BYTES;
  static constexpr int SMEM_BYTES = OFF_BAR + 1024 + 256;
  static constexpr int NUM_THREADS = 64 + 32 * EW;
  static_assert(SMEM_BYTES + 256 <= 232448, "shared memory of a CTA");
};
constexpr int GROUP_M = 8;
constexpr int MAX_PROBLEMS = 8;

// epi selects the epilogue of a problem:
//   0  C = acc (+ C when accumulate)
//   1  SwiGLU forward: B is a fused [2 * half, K] gate | up weight.  Tile tn holds 128 gate columns
//      (accumulator columns 0..127) and the 128 up columns of the same index (128..255): both go to
//      C [M, 2 * half] as usual (the backward needs them; a null C is not stored) and silu(g) * u goes to C2 [M, half].
//   2  SwiGLU backward: acc is dh [M, half] of the down projection; the epilogue reads g | u from
//      C2 [M, 2 * half] and writes dg | du to C [M, 2 * half]; dh itself is never stored.
//   4  C = acc with its first columns rotated (RopeArgs).
struct Problem {
  const bf16* old;      // what the epilogue reads: C when accumulate, C2 (g | u) with epi 2
  long long ld_old;
  bf16* C;
  long long ldc;
  int M, N, K;
  int a_mn, b_mn, accumulate;
  int tiles_m, tiles_n, num_kb;
  int epi, half;
  int keep;             // epi 1: C is stored
};

template <int NP>
struct GroupedParams {
  CUtensorMap ta[NP];
  CUtensorMap tb[NP];
  CUtensorMap tc[NP][3];      // where the epilogue stores with TMA: C; C's gate columns, its up columns, C2 (epi 1)
  Problem prob[NP];
  RopeArgs rope;
  const int* offsets;   // [grid + 1] first item of every CTA
  const int* items;     // (problem << 24) | tile index inside the problem
};

__device__ __forceinline__ void tile_coords(int t, const Problem& p, int& tm, int& tn) {
  const int group_size = GROUP_M * p.tiles_n;
  const int group = t / group_size;
  const int first_m = group * GROUP_M;
  const int gsz = min(p.tiles_m - first_m, GROUP_M);
  const int in_group = t - group * group_size;
  tm = first_m + in_group % gsz;
  tn = in_group / gsz;
}

__device__ __forceinline__ void give_up(volatile int* abort_flag, unsigned where) {
  *abort_flag = 1;
  atomicExch(&g_grp_status[0], 1u);
  atomicExch(&g_grp_status[1], where);
}

// One tile of the producer / of the MMA issuer, specialised on the operand majors: with the majors
// as compile-time constants every descriptor field and the number of TMA boxes is a constant (with
// run-time majors the producer issued predicated-off TMA instructions for the branch not taken and
// the tensor pipe lost a fifth of its activity), although the tile itself comes from a list in memory.
// A CTA of a pair loads its own part (m0, n0 are its first row of A and of B) and signals the leader's barrier,
// which expects the bytes of both.
template <int CG>
__device__ __forceinline__ void load_box(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  if constexpr (CG == 2) bw::tma_load_2d_pair(dst, map, x, y, bar);
  else bw::tma_load_2d(dst, map, x, y, bar);
}
template <typename C, int CG, bool A_MN, bool B_MN>
__device__ __forceinline__ bool produce_tile(const CUtensorMap* ta, const CUtensorMap* tb, int m0, int n0, int num_kb,
                                             uint32_t smem_base, uint32_t bar_base, int& stage, uint32_t& phase,
                                             volatile int* abort_flag, bool leader, int k_base = 0, int b_split = 0) {
  for (int kb = 0; kb < num_kb; kb++) {
    if (!bw::mbar_wait(bar_base + 8u * (C::STAGES + stage), phase ^ 1u, abort_flag)) return false;
    uint32_t fb = bar_base + 8u * stage;
    if (CG == 1 || leader) bw::mbar_expect_tx(fb, CG * C::STAGE_BYTES);
    if (CG == 2) fb = bw::leader_bar(fb);
    const uint32_t sa = smem_base + stage * C::STAGE_BYTES;
    const uint32_t sb = sa + A_BYTES;
    const int k0 = k_base + kb * BK;
    if (!A_MN) {
      load_box<CG>(sa, ta, k0, m0, fb);                                                              // box {64 k, 128 m}
    } else {
#pragma unroll
      for (int j = 0; j < BM / 64; j++) load_box<CG>(sa + j * 8192, ta, m0 + 64 * j, k0, fb);        // box {64 m, 64 k}
    }
    if (!B_MN) {
      load_box<CG>(sb, tb, k0, n0, fb);                                                              // box {64 k, 128 n}
      if (CG == 1)                               // second box: the next 128 rows, or (SwiGLU) the up rows b_split + n0..
        load_box<CG>(sb + (BN / 2) * BK * 2, tb, k0, n0 + (b_split > 0 ? b_split : BN / 2), fb);
    } else {
#pragma unroll
      for (int j = 0; j < BN / CG / 64; j++) load_box<CG>(sb + j * 8192, tb, n0 + 64 * j, k0, fb);   // box {64 n, 64 k}
    }
    if (++stage == C::STAGES) { stage = 0; phase ^= 1u; }
  }
  return true;
}

template <typename C, int CG, bool A_MN, bool B_MN>
__device__ __forceinline__ bool mma_tile(uint32_t d_tmem, int num_kb, uint32_t smem_base, uint32_t bar_base, int& stage,
                                         uint32_t& phase, volatile int* abort_flag) {
  constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((A_MN ? 1u : 0u) << 15) | ((B_MN ? 1u : 0u) << 16) |
                             ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(BM * CG >> 4) << 24);
  constexpr uint32_t a_lbo = A_MN ? 8192u : 16u, b_lbo = B_MN ? 8192u : 16u;
  constexpr uint32_t a_kstep = A_MN ? 2048u : 32u, b_kstep = B_MN ? 2048u : 32u;   // bytes per K=16 slice
  for (int kb = 0; kb < num_kb; kb++) {
    if (!bw::mbar_wait(bar_base + 8u * stage, phase, abort_flag)) return false;
    bw::fence_after();
    const uint32_t sa = smem_base + stage * C::STAGE_BYTES;
    const uint32_t sb = sa + A_BYTES;
#pragma unroll
    for (int k = 0; k < BK / 16; k++) {
      const uint64_t ad = bw::make_desc(sa + k * a_kstep, a_lbo, 1024u);
      const uint64_t bd = bw::make_desc(sb + k * b_kstep, b_lbo, 1024u);
      if constexpr (CG == 2) bw::umma_bf16_pair(d_tmem, ad, bd, idesc, (kb | k) ? 1u : 0u);
      else bw::umma_bf16(d_tmem, ad, bd, idesc, (kb | k) ? 1u : 0u);
    }
    // frees this smem stage (of both CTAs) when the MMAs have read it
    if constexpr (CG == 2) bw::umma_commit_pair(bar_base + 8u * (C::STAGES + stage));
    else bw::umma_commit(bar_base + 8u * (C::STAGES + stage));
    if (++stage == C::STAGES) { stage = 0; phase ^= 1u; }
  }
  return true;
}

// ---- epilogue of a warp: 32 rows x 256 or 128 columns of an accumulator ------------------------------------
// Columns pass through one of the warp's 4 KB staging buffers (swizzled, a row per lane), 64 at a time.  What is only written leaves by a TMA store, which ends at
// the matrix's last row and column.  Where the epilogue also reads (the old C, or g | u), steps of 32 columns: four lanes read and write a row's part, the
// loads a step ahead of their use, and rows turn into lanes and back in the buffer.  A row per lane read and written straight from memory is 32
// lines for every 16 bytes per lane, and kept the load/store unit busy for as long as a main loop of K = 2048 takes (epi 2).  The same
// launches with that form / this, us: 562 / 487, 696 / 545, 1082 / 1033, and 250 / 245 for the down projection; of 1000 x 768 -> 2048: 12.4 / 11.2, 22.1 / 16.6
// (SwiGLU backward), 28.9 / 26.5.  (With TMA stores, whose fence waits for loads in flight, the SwiGLU backward took 579; with
// stores from whole lines of the buffer in their place the forward 505.)
struct Out {
  const CUtensorMap* map;
  const bf16* old;     // EPI 2, 3: what is read and where the result goes
  long long ld_old;
  bf16* out;
  long long ld_out;
  int row0, rows;      // the warp's first row, rows of the matrix
  int c0, cols;        // the warp's first column, columns (of one half, with an activation)
  bool keep;           // EPI 1: g and u are stored
  const RopeArgs* rope;
};

// EPI as in Problem; 3: C = acc + C.  taddr: the warp's first column (EPI 1: of g).  ready() waits for the accumulator, release() gives its columns back.
// `turn`: the buffer that is next, kept over the tiles.
template <int EPI, int NBUF, int EW, typename Ready, typename Release>
__device__ __forceinline__ bool store_tile(const Out& o, uint32_t taddr, uint8_t* stg, int& turn, int lane, Ready ready, Release release) {
  constexpr int COLS = BN * 4 / EW;                                   // of the warp (EPI 1: half of them of g, half of u)
  if (o.c0 >= o.cols) {
    if (!ready()) return false;
    release();
    return true;
  }
  if constexpr (EPI == 2 || EPI == 3) {
    const int lr = lane >> 2, lc = (lane & 3) * 8;                    // memory accesses: row (of every eight), column
    uint8_t* const stg2 = stg + STG_BYTES / 2;
    // 16-byte piece c of row r: rows are 64 B apart, no bank twice for eight rows' one piece or two rows' four
    auto at = [&](uint8_t* buf, int r, int c) { return reinterpret_cast<uint4*>(buf + r * 64 + ((c ^ ((r >> 1) & 3)) << 4)); };
    uint4 old[4], old2[EPI == 2 ? 4 : 1];
    auto inside = [&](int i, int c) { return o.row0 + 8 * i + lr < o.rows && o.c0 + c * 32 + lc < o.cols; };
    auto fetch = [&](int c) {
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const bf16* from = o.old + (size_t)(o.row0 + 8 * i + lr) * o.ld_old + o.c0 + c * 32 + lc;
        const bool in = inside(i, c);
        old[i] = in ? *reinterpret_cast<const uint4*>(from) : make_uint4(0, 0, 0, 0);
        if constexpr (EPI == 2) old2[i] = in ? *reinterpret_cast<const uint4*>(from + o.cols) : make_uint4(0, 0, 0, 0);
      }
    };
    fetch(0);
    if (!ready()) return false;
    if (lane == 0) bw::bulk_wait_read_but<0>();                       // (stores of another kind of tile)
    __syncwarp();
#pragma unroll 1
    for (int c = 0; c < COLS / 32; c++) {
      const bool last = c == COLS / 32 - 1 || o.c0 + (c + 1) * 32 >= o.cols;
#pragma unroll
      for (int i = 0; i < 4; i++) {
        *at(stg, 8 * i + lr, lane & 3) = old[i];
        if constexpr (EPI == 2) *at(stg2, 8 * i + lr, lane & 3) = old2[i];
      }
      if (!last) fetch(c + 1);
      uint32_t r[32];
      bw::tmem_ld32(taddr + c * 32, r);
      bw::tmem_ld_wait();
      if (last) release();
      __syncwarp();
#pragma unroll
      for (int g = 0; g < 4; g++) {
        float f[8], fg[8];
#pragma unroll
        for (int i = 0; i < 8; i++) f[i] = __uint_as_float(r[g * 8 + i]);
        unpack8(*at(stg, lane, g), fg);
        if constexpr (EPI == 2) {
          const bw::f32x2 one = bw::pack2(1.f, 1.f), minus = bw::pack2(-1.f, -1.f);
          float fu[8];
          unpack8(pack8(f), f);                                       // the value a stored bf16 dh would have had
          unpack8(*at(stg2, lane, g), fu);
#pragma unroll
          for (int i = 0; i < 8; i += 2) {
            const bw::f32x2 d = bw::pack2(f[i], f[i + 1]), gg = bw::pack2(fg[i], fg[i + 1]), uu = bw::pack2(fu[i], fu[i + 1]);
            float a, b;
            bw::unpack2(bw::add2(one, bw::pack2(__expf(-fg[i]), __expf(-fg[i + 1]))), a, b);
            const bw::f32x2 sig = bw::pack2(1.f / a, 1.f / b);
            const bw::f32x2 slope = bw::fma2(gg, bw::fma2(sig, minus, one), one);
            bw::unpack2(bw::mul2(bw::mul2(bw::mul2(d, uu), sig), slope), f[i], f[i + 1]);       // dg
            bw::unpack2(bw::mul2(bw::mul2(d, gg), sig), fu[i], fu[i + 1]);                      // du
          }
          *at(stg2, lane, g) = pack8(fu);
        } else {
#pragma unroll
          for (int i = 0; i < 8; i++) f[i] += fg[i];
        }
        *at(stg, lane, g) = pack8(f);
      }
      __syncwarp();
#pragma unroll
      for (int i = 0; i < 4; i++) {
        bf16* to = o.out + (size_t)(o.row0 + 8 * i + lr) * o.ld_out + o.c0 + c * 32 + lc;
        if (inside(i, c)) {
          *reinterpret_cast<uint4*>(to) = *at(stg, 8 * i + lr, lane & 3);
          if constexpr (EPI == 2) *reinterpret_cast<uint4*>(to + o.cols) = *at(stg2, 8 * i + lr, lane & 3);
        }
      }
      __syncwarp();
      if (last) break;
    }
    return true;
  }
  auto store = [&](const uint4* rows8, const CUtensorMap* map, int col) {      // a lane's row of 64 columns
    if (lane == 0) bw::bulk_wait_read_but<NBUF - 1>();                // the last store from this buffer has read it
    __syncwarp();
    uint8_t* buf = stg + turn * STG_BYTES;
    if (NBUF > 1) turn ^= 1;
#pragma unroll
    for (int g = 0; g < 8; g++) *reinterpret_cast<uint4*>(buf + bw::sw128_off(lane, g)) = rows8[g];
    bw::fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) {
      if (o.row0 < o.rows) bw::tma_store_2d(map, bw::smem_u32(buf), col, o.row0);
      bw::bulk_commit();
    }
  };
  if (!ready()) return false;
  if constexpr (EPI == 1) {
    // g and u are stored, and silu(g) * u computed from the ROUNDED values (what a separate pass over the stored
    // matrix would see, and what the backward recomputes from)
#pragma unroll 1
    for (int c = 0; c < COLS / 128; c++) {
      const int col = o.c0 + c * 64;
      const bool last = c == COLS / 128 - 1 || col + 64 >= o.cols;
      uint4 pg[8], pu[8];
      auto take32 = [&](uint32_t from, uint4* p) {
        float f[32];
        bw::tmem_ld32(from, reinterpret_cast<uint32_t*>(f));
        bw::tmem_ld_wait();
#pragma unroll
        for (int g = 0; g < 4; g++) p[g] = pack8(f + g * 8);
      };
      take32(taddr + c * 64, pg);
      take32(taddr + c * 64 + 32, pg + 4);
      take32(taddr + BN / 2 + c * 64, pu);
      take32(taddr + BN / 2 + c * 64 + 32, pu + 4);
      if (last) release();
      if (o.keep) {
        store(pg, o.map, col);
        store(pu, o.map + 1, col);
      }
#pragma unroll
      for (int g = 0; g < 8; g++) {
        float fg[8], fu[8];
        unpack8(pg[g], fg);
        unpack8(pu[g], fu);
#pragma unroll
        for (int i = 0; i < 8; i++) fg[i] = fg[i] / (1.f + __expf(-fg[i])) * fu[i];
        pg[g] = pack8(fg);
      }
      store(pg, o.map + 2, col);
      if (last) break;
    }
  } else {
    const int pos = EPI == 4 && o.row0 + lane < o.rows ? rope_position(*o.rope, o.row0 + lane) : 0;
#pragma unroll 1
    for (int c = 0; c < COLS / 64; c++) {
      const int col = o.c0 + c * 64;
      const bool last = c == COLS / 64 - 1 || col + 64 >= o.cols;
      float f[64];
      uint4 p[8];
      bw::tmem_ld32(taddr + c * 64, reinterpret_cast<uint32_t*>(f));
      bw::tmem_ld32(taddr + c * 64 + 32, reinterpret_cast<uint32_t*>(f) + 32);
      bw::tmem_ld_wait();
      if (last) release();
#pragma unroll
      for (int g = 0; g < 8; g++) {
        p[g] = pack8(f + g * 8);
        if constexpr (EPI == 4) {
          if (col + g * 8 < o.rope->cols) {
            float v[8], cs[8];
            unpack8(p[g], v);                                         // the values a stored C would have
            rope_load8(*o.rope, pos, col + g * 8, cs);
            rope_rotate8(cs, v);
            p[g] = pack8(v);
          }
        }
      }
      store(p, o.map, col);
      if (last) break;
    }
  }
  return true;
}

template <int CG, int EW, int NP>
__global__ void __launch_bounds__(Cfg<CG, EW>::NUM_THREADS, 1) gemm_grouped_kernel(const __grid_constant__ GroupedParams<NP> gp) {
  using CF = Cfg<CG, EW>;
  constexpr int STAGES = CF::STAGES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + CF::OFF_BAR);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 4);
  __shared__ int s_abort[2];     // {abort, extra wait in ms}: see bw::mbar_wait

  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0);      // (uniform over the warp)
  const int lane = threadIdx.x & 31;
  const uint32_t smem_base = bw::smem_u32(smem);
  const uint32_t bar_base = bw::smem_u32(bars);
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (STAGES + s); };
  auto tfull_bar = [&](int a) { return bar_base + 8u * (2 * STAGES + a); };
  auto tempty_bar = [&](int a) { return bar_base + 8u * (2 * STAGES + 2 + a); };
  const int worker = (int)blockIdx.x / CG;                       // a CTA, or a pair of CTAs that walks one list
  const int rank = CG == 2 ? (int)bw::cluster_ctarank() : 0;      // 0 = leader: issues the MMAs of the pair
  const int item_begin = gp.offsets[worker], item_end = gp.offsets[worker + 1];

  if (threadIdx.x == 0) {
    s_abort[0] = 0;
    s_abort[1] = 0;
    for (int s = 0; s < STAGES; s++) {
      bw::mbar_init(full_bar(s), 1);
      bw::mbar_init(empty_bar(s), 1);
    }
    for (int a = 0; a < 2; a++) {
      bw::mbar_init(tfull_bar(a), 1);
      bw::mbar_init(tempty_bar(a), EW * CG);
    }
    bw::mbar_init_fence();
  }
  if (warp == 1) {
    if constexpr (CG == 2) bw::tmem_alloc_pair(bw::smem_u32(tmem_slot), 512);
    else bw::tmem_alloc(bw::smem_u32(tmem_slot), 512);
  }
  bw::fence_before();
  __syncthreads();
  if constexpr (CG == 2) bw::cluster_sync();      // the peer's barriers exist before anything signals them
  bw::fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  volatile int* abort_flag = s_abort;
  // (No grid_go(): the next kernel's CTAs would crowd into the SMs that are done first.)
  grid_wait();

  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    if (bw::elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      int next_item = item_begin < item_end ? gp.items[item_begin] : 0;
      for (int it = item_begin; it < item_end && ok; it++) {
        const int item = next_item;
        if (it + 1 < item_end) next_item = gp.items[it + 1];      // in flight while this tile streams
        const int pi = item >> 24;
        const CUtensorMap* ta = &gp.ta[pi];
        const CUtensorMap* tb = &gp.tb[pi];
        int tm, tn;
        tile_coords(item & 0xFFFFFF, gp.prob[pi], tm, tn);
        const int split = gp.prob[pi].epi == 1 ? gp.prob[pi].half : 0;
        // first row of A and of B this CTA loads.  SwiGLU tiles: 128 gate rows and the up rows of the same
        // index (a pair's leader loads the former, its peer the latter)
        const int m0 = (tm * CG + rank) * BM;
        const int n0 = split ? tn * (BN / 2) + (CG == 2 ? rank * split : 0) : tn * BN + rank * (BN / 2);
        const int num_kb = gp.prob[pi].num_kb;
        switch (gp.prob[pi].a_mn * 2 + gp.prob[pi].b_mn) {
          case 0: ok = produce_tile<CF, CG, false, false>(ta, tb, m0, n0, num_kb, smem_base, bar_base, stage, phase, abort_flag, rank == 0, 0, split); break;
          case 1: ok = produce_tile<CF, CG, false, true>(ta, tb, m0, n0, num_kb, smem_base, bar_base, stage, phase, abort_flag, rank == 0); break;
          case 2: ok = produce_tile<CF, CG, true, false>(ta, tb, m0, n0, num_kb, smem_base, bar_base, stage, phase, abort_flag, rank == 0, 0, split); break;
          default: ok = produce_tile<CF, CG, true, true>(ta, tb, m0, n0, num_kb, smem_base, bar_base, stage, phase, abort_flag, rank == 0); break;
        }
        if (!ok) give_up(abort_flag, 1u);
      }
      // the leader's MMAs release this CTA's stages: all releases have arrived before the CTA may exit
      if (CG == 2)
        for (int s = 0; s < STAGES && ok; s++) {
          ok = bw::mbar_wait(empty_bar(stage), phase ^ 1u, abort_flag);
          if (++stage == STAGES) { stage = 0; phase ^= 1u; }
        }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer ------------------------------
    if (rank == 0 && bw::elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      int n = 0;
      int next_item = item_begin < item_end ? gp.items[item_begin] : 0;
      for (int it = item_begin; it < item_end && ok; it++, n++) {
        const int pi = next_item >> 24;
        if (it + 1 < item_end) next_item = gp.items[it + 1];
        const int num_kb = gp.prob[pi].num_kb;
        const int majors = gp.prob[pi].a_mn * 2 + gp.prob[pi].b_mn;
        const int acc = n & 1;
        const uint32_t acc_phase = (uint32_t)(n >> 1) & 1u;
        if (!bw::mbar_wait(tempty_bar(acc), acc_phase ^ 1u, abort_flag)) { give_up(abort_flag, 2u); ok = false; break; }
        bw::fence_after();
        const uint32_t d_tmem = tmem_base + (uint32_t)acc * BN;
        switch (majors) {
          case 0: ok = mma_tile<CF, CG, false, false>(d_tmem, num_kb, smem_base, bar_base, stage, phase, abort_flag); break;
          case 1: ok = mma_tile<CF, CG, false, true>(d_tmem, num_kb, smem_base, bar_base, stage, phase, abort_flag); break;
          case 2: ok = mma_tile<CF, CG, true, false>(d_tmem, num_kb, smem_base, bar_base, stage, phase, abort_flag); break;
          default: ok = mma_tile<CF, CG, true, true>(d_tmem, num_kb, smem_base, bar_base, stage, phase, abort_flag); break;
        }
        if (!ok) give_up(abort_flag, 3u);
        else if constexpr (CG == 2) bw::umma_commit_pair(tfull_bar(acc));          // accumulator complete
        else bw::umma_commit(tfull_bar(acc));
      }
    }
  } else {
    // ------------------------------ epilogue ------------------------------
    const int quad = warp & 3, part = (warp - 2) >> 2;
    uint8_t* stg = smem + CF::OFF_STG + (warp - 2) * CF::NBUF * STG_BYTES;
    int n = 0, turn = 0;
    int next_item = item_begin < item_end ? gp.items[item_begin] : 0;
    for (int it = item_begin; it < item_end; it++, n++) {
      const int item = next_item;
      if (it + 1 < item_end) next_item = gp.items[it + 1];
      const int pi = item >> 24;
      int tm, tn;
      tile_coords(item & 0xFFFFFF, gp.prob[pi], tm, tn);
      const Problem& pr = gp.prob[pi];
      const int acc = n & 1;
      const uint32_t acc_phase = (uint32_t)(n >> 1) & 1u;
      const Out out{gp.tc[pi], pr.old, pr.ld_old, pr.C, pr.ldc, (tm * CG + rank) * BM + quad * 32, pr.M,
                    tn * (pr.epi == 1 ? BN / 2 : BN) + part * (pr.epi == 1 ? BN / 4 : BN / 2), pr.epi == 1 || pr.epi == 2 ? pr.half : pr.N, pr.keep != 0, &gp.rope};
      const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(acc * BN + part * (pr.epi == 1 ? BN / 4 : BN / 2));
      auto ready = [&]() {
        if (!bw::mbar_wait(tfull_bar(acc), acc_phase, abort_flag)) return false;
        bw::fence_after();
        return true;
      };
      auto release = [&]() {
        bw::fence_before();
        __syncwarp();
        if (lane == 0) {
          if constexpr (CG == 2) bw::mbar_arrive_leader(tempty_bar(acc));
          else bw::mbar_arrive(tempty_bar(acc));
        }
      };
      bool ok;
      switch (pr.epi == 0 && pr.accumulate ? 3 : pr.epi) {
        case 0: ok = store_tile<0, CF::NBUF, EW>(out, taddr, stg, turn, lane, ready, release); break;
        case 1: ok = store_tile<1, CF::NBUF, EW>(out, taddr, stg, turn, lane, ready, release); break;
        case 2:
          if constexpr (EW == 8) ok = store_tile<2, CF::NBUF, EW>(out, taddr, stg, turn, lane, ready, release);      // (launches with it take eight)
          else ok = false;
          break;
        case 4: ok = store_tile<4, CF::NBUF, EW>(out, taddr, stg, turn, lane, ready, release); break;
        default: ok = store_tile<3, CF::NBUF, EW>(out, taddr, stg, turn, lane, ready, release); break;
      }
      if (!ok) { give_up(abort_flag, 4u); break; }
    }
    if (lane == 0) bw::bulk_wait_read_but<0>();        // nothing reads shared memory after the CTA's end
  }

  bw::fence_before();
  __syncthreads();
  if constexpr (CG == 2) bw::cluster_sync();      // nothing of the pair is in flight in either CTA
  if (warp == 1) {
    bw::fence_after();
    if constexpr (CG == 2) bw::tmem_dealloc_pair(tmem_base, 512);
    else bw::tmem_dealloc(tmem_base, 512);
  }
}

// ---- ragged variant: row segments whose sizes live in device memory --------------------------------
// The per-expert GEMMs of a MoE layer.  One activation buffer [cap, K] holds the rows of all local
// experts, expert e in rows [seg[e], seg[e] + seg[LE + e]); every segment starts on a multiple of
// 128 rows and the rows between a segment's end and the next multiple of 128 are zero.  Offsets and
// counts are written by the planning kernel of the token exchange (moe.cu) and are never read on
// the host: every role of every CTA derives the same tile list from them.
//   mode 0   C[rows of e, N] = A[rows of e, K] . op(B_e)^T           (forward, data gradient)
//            all tiles cost the same, so CTA c simply takes tiles c, c + grid, ...
//   mode 1   C_e[Nw, Kw] (+)= A[rows of e, Nw]^T . B[rows of e, Kw]  (weight gradient; the reduction
//            runs over the rows of the segment, in 64-row steps, padding rows contribute zeros)
// Before its first load the producer can wait (bounded) for an arrival word: the rows are pushed
// into A by other GPUs.
struct RaggedParams {
  CUtensorMap ta;                      // mode 0: [cap, K] K-major;  mode 1: [cap, Nw] as MN-major A
  CUtensorMap tb[MAX_PROBLEMS];        // mode 0: B_e;               mode 1: tb[0] = [cap, Kw] as MN-major B
  CUtensorMap tc[MAX_PROBLEMS];        // mode 0: tc[0..2] as in GroupedParams, of matrices of cap rows;  mode 1: C_e
  bf16* C[MAX_PROBLEMS];               // mode 0: C[0];  mode 1: C_e
  long long ldc;
  const bf16* old;                     // mode 0, epi 2: g | u
  long long ld_old;
  int epi, half, keep;                 // (keep: see Problem)
  const int* seg;
  int LE, M_w, N, K, b_mn, mode, accumulate, cap;
  int tiles_n, tiles_m_w, num_kb;
  const unsigned int* wait_flag;
  unsigned int wait_target;
  unsigned long long wait_ns;
};

struct RaggedTile { int e, m0, n0, num_kb, k_base; };

// Tile `t` of the launch, or e < 0 past the end.  seg_* are the CTA's shared copies of the table.
template <int CG>
__device__ __forceinline__ RaggedTile ragged_tile(int t, const RaggedParams& rp, const int* s_off, const int* s_tiles) {
  RaggedTile r;
  r.e = -1; r.m0 = r.n0 = r.num_kb = r.k_base = 0;
  if (rp.mode == 0) {
    for (int e = 0; e < rp.LE; e++) {
      const int nt = s_tiles[e] * rp.tiles_n;
      if (t < nt) {
        Problem pr;
        pr.tiles_m = s_tiles[e]; pr.tiles_n = rp.tiles_n;
        int tm, tn;
        tile_coords(t, pr, tm, tn);
        r.e = e; r.m0 = s_off[e] + tm * BM * CG; r.n0 = tn * (rp.epi == 1 ? BN / 2 : BN); r.num_kb = rp.num_kb;
        return r;
      }
      t -= nt;
    }
  } else {
    const int per = rp.tiles_m_w * rp.tiles_n;
    const int e = t / per;
    if (e < rp.LE) {
      const int tt = t - e * per;
      r.e = e; r.m0 = (tt % rp.tiles_m_w) * BM * CG; r.n0 = (tt / rp.tiles_m_w) * BN;
      r.num_kb = s_tiles[e];              // 64-row steps over the segment
      r.k_base = s_off[e];
    }
  }
  return r;
}

template <int CG, int EW>
__global__ void __launch_bounds__(Cfg<CG, EW>::NUM_THREADS, 1) gemm_ragged_kernel(const __grid_constant__ RaggedParams rp) {
  using CF = Cfg<CG, EW>;
  constexpr int STAGES = CF::STAGES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + CF::OFF_BAR);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 4);
  __shared__ int s_abort[2];     // {abort, extra wait in ms}: see bw::mbar_wait
  __shared__ int s_off[MAX_PROBLEMS], s_tiles[MAX_PROBLEMS], s_end[MAX_PROBLEMS];

  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0);      // (uniform over the warp)
  const int lane = threadIdx.x & 31;
  const uint32_t smem_base = bw::smem_u32(smem);
  const uint32_t bar_base = bw::smem_u32(bars);
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (STAGES + s); };
  auto tfull_bar = [&](int a) { return bar_base + 8u * (2 * STAGES + a); };
  auto tempty_bar = [&](int a) { return bar_base + 8u * (2 * STAGES + 2 + a); };

  const int worker = (int)blockIdx.x / CG, workers = (int)gridDim.x / CG;
  const int rank = CG == 2 ? (int)bw::cluster_ctarank() : 0;      // 0 = leader: issues the MMAs of the pair

  if (threadIdx.x == 0) {
    s_abort[0] = 0;
    s_abort[1] = rp.wait_flag ? bw::wait_extra_ms(rp.wait_ns) : 0;
    for (int s = 0; s < STAGES; s++) {
      bw::mbar_init(full_bar(s), 1);
      bw::mbar_init(empty_bar(s), 1);
    }
    for (int a = 0; a < 2; a++) {
      bw::mbar_init(tfull_bar(a), 1);
      bw::mbar_init(tempty_bar(a), EW * CG);
    }
    bw::mbar_init_fence();
  }
  if (warp == 1) {
    if constexpr (CG == 2) bw::tmem_alloc_pair(bw::smem_u32(tmem_slot), 512);
    else bw::tmem_alloc(bw::smem_u32(tmem_slot), 512);
  }
  grid_wait();
  if (threadIdx.x < rp.LE) {
    // segment table -> offsets and tile (mode 0: 128-row tiles) / step (mode 1: 64-row steps) counts,
    // clamped so that no coordinate can pass the end of the buffer
    int off = rp.seg[threadIdx.x], cnt = rp.seg[rp.LE + threadIdx.x];
    if (off < 0 || off > rp.cap) { off = 0; cnt = 0; }
    if (cnt < 0) cnt = 0;
    if (off + cnt > rp.cap) cnt = rp.cap - off;
    s_off[threadIdx.x] = off;
    s_tiles[threadIdx.x] = rp.mode == 0 ? (cnt + BM * CG - 1) / (BM * CG) : (cnt + BK - 1) / BK;
    s_end[threadIdx.x] = min(off + (cnt + BM - 1) / BM * BM, rp.cap);      // (the second CTA's rows may be the next segment's)
  }
  bw::fence_before();
  __syncthreads();
  if constexpr (CG == 2) bw::cluster_sync();      // the peer's barriers exist before anything signals them
  bw::fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  volatile int* abort_flag = s_abort;

  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    if (bw::elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      if (rp.wait_flag) {
        // the rows of A are pushed by other GPUs: acquire the arrival word, then order their
        // generic-proxy writes before the TMA (async proxy) reads
        if (!lbcomm::flag_wait_ge(rp.wait_flag, rp.wait_target, rp.wait_ns)) { give_up(abort_flag, 11u); ok = false; }
        asm volatile("fence.proxy.async;" ::: "memory");
      }
      for (int t = worker; ok; t += workers) {
        const RaggedTile rt = ragged_tile<CG>(t, rp, s_off, s_tiles);
        if (rt.e < 0) break;
        if (rt.num_kb == 0) continue;
        const int split = rp.epi == 1 ? rp.half : 0;
        // this CTA's first rows of A and of B (see gemm_grouped_kernel)
        const int m0 = rt.m0 + rank * BM, n0 = rt.n0 + (CG == 2 ? rank * (split ? split : BN / 2) : 0);
        if (rp.mode == 0) {
          if (!rp.b_mn) ok = produce_tile<CF, CG, false, false>(&rp.ta, &rp.tb[rt.e], m0, n0, rt.num_kb, smem_base, bar_base, stage, phase, abort_flag, rank == 0, 0, split);
          else          ok = produce_tile<CF, CG, false, true>(&rp.ta, &rp.tb[rt.e], m0, n0, rt.num_kb, smem_base, bar_base, stage, phase, abort_flag, rank == 0);
        } else {
          ok = produce_tile<CF, CG, true, true>(&rp.ta, &rp.tb[0], m0, n0, rt.num_kb, smem_base, bar_base, stage, phase, abort_flag, rank == 0, rt.k_base);
        }
        if (!ok) give_up(abort_flag, 1u);
      }
      // the leader's MMAs release this CTA's stages: all releases have arrived before the CTA may exit
      if (CG == 2)
        for (int s = 0; s < STAGES && ok; s++) {
          ok = bw::mbar_wait(empty_bar(stage), phase ^ 1u, abort_flag);
          if (++stage == STAGES) { stage = 0; phase ^= 1u; }
        }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer ------------------------------
    if (rank == 0 && bw::elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      int n = 0;
      for (int t = worker; ok; t += workers) {
        const RaggedTile rt = ragged_tile<CG>(t, rp, s_off, s_tiles);
        if (rt.e < 0) break;
        if (rt.num_kb == 0) continue;
        const int acc = n & 1;
        const uint32_t acc_phase = (uint32_t)(n >> 1) & 1u;
        if (!bw::mbar_wait(tempty_bar(acc), acc_phase ^ 1u, abort_flag)) { give_up(abort_flag, 2u); ok = false; break; }
        bw::fence_after();
        const uint32_t d_tmem = tmem_base + (uint32_t)acc * BN;
        if (rp.mode == 0) {
          if (!rp.b_mn) ok = mma_tile<CF, CG, false, false>(d_tmem, rt.num_kb, smem_base, bar_base, stage, phase, abort_flag);
          else          ok = mma_tile<CF, CG, false, true>(d_tmem, rt.num_kb, smem_base, bar_base, stage, phase, abort_flag);
        } else {
          ok = mma_tile<CF, CG, true, true>(d_tmem, rt.num_kb, smem_base, bar_base, stage, phase, abort_flag);
        }
        if (!ok) give_up(abort_flag, 3u);
        else if constexpr (CG == 2) bw::umma_commit_pair(tfull_bar(acc));
        else bw::umma_commit(tfull_bar(acc));
        n++;
      }
    }
  } else {
    // ------------------------------ epilogue ------------------------------
    const int quad = warp & 3, part = (warp - 2) >> 2;
    uint8_t* stg = smem + CF::OFF_STG + (warp - 2) * CF::NBUF * STG_BYTES;
    int n = 0, turn = 0;
    for (int t = worker;; t += workers) {
      const RaggedTile rt = ragged_tile<CG>(t, rp, s_off, s_tiles);
      if (rt.e < 0) break;
      if (rt.num_kb == 0) {
        // an expert without rows: its weight gradient is zero (nothing to add when accumulating)
        const int row = rt.m0 + rank * BM + quad * 32 + lane;
        if (rp.mode == 1 && !rp.accumulate && row < rp.M_w)
          for (int c = rt.n0 + part * (BN / 2); c < rt.n0 + (EW == 4 ? BN : (part + 1) * (BN / 2)) && c < rp.N; c += 8)
            *reinterpret_cast<uint4*>(rp.C[rt.e] + (size_t)row * rp.ldc + c) = make_uint4(0, 0, 0, 0);
        continue;
      }
      const int acc = n & 1;
      const uint32_t acc_phase = (uint32_t)(n >> 1) & 1u;
      const bool wgrad = rp.mode == 1;
      // (mode 0 writes whole 128-row tiles: padding rows are zeros)
      const Out out{wgrad ? &rp.tc[rt.e] : rp.tc, wgrad ? rp.C[rt.e] : rp.old, wgrad ? rp.ldc : rp.ld_old, wgrad ? rp.C[rt.e] : rp.C[0], rp.ldc, rt.m0 + rank * BM + quad * 32, wgrad ? rp.M_w : s_end[rt.e],
                    rt.n0 + part * (rp.epi == 1 ? BN / 4 : BN / 2), rp.epi ? rp.half : rp.N, rp.keep != 0, nullptr};
      const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(acc * BN + part * (rp.epi == 1 ? BN / 4 : BN / 2));
      auto ready = [&]() {
        if (!bw::mbar_wait(tfull_bar(acc), acc_phase, abort_flag)) return false;
        bw::fence_after();
        return true;
      };
      auto release = [&]() {
        bw::fence_before();
        __syncwarp();
        if (lane == 0) {
          if constexpr (CG == 2) bw::mbar_arrive_leader(tempty_bar(acc));
          else bw::mbar_arrive(tempty_bar(acc));
        }
      };
      bool ok;
      switch (wgrad && rp.accumulate ? 3 : rp.epi) {
        case 0: ok = store_tile<0, CF::NBUF, EW>(out, taddr, stg, turn, lane, ready, release); break;
        case 1: ok = store_tile<1, CF::NBUF, EW>(out, taddr, stg, turn, lane, ready, release); break;
        case 2:
          if constexpr (EW == 8) ok = store_tile<2, CF::NBUF, EW>(out, taddr, stg, turn, lane, ready, release);      // (launches with it take eight)
          else ok = false;
          break;
        default: ok = store_tile<3, CF::NBUF, EW>(out, taddr, stg, turn, lane, ready, release); break;
      }
      if (!ok) { give_up(abort_flag, 4u); break; }
      n++;
    }
    if (lane == 0) bw::bulk_wait_read_but<0>();        // nothing reads shared memory after the CTA's end
  }

  bw::fence_before();
  __syncthreads();
  if constexpr (CG == 2) bw::cluster_sync();      // nothing of the pair is in flight in either CTA
  if (warp == 1) {
    bw::fence_after();
    if constexpr (CG == 2) bw::tmem_dealloc_pair(tmem_base, 512);
    else bw::tmem_dealloc(tmem_base, 512);
  }
}

// ---- host side: static schedule, cached per (device, shapes) -------------------------------------
struct Schedule {
  int split = 0;      // parts of K of a launch that the split form takes (gemm_split.cu; nothing else is set then), or 0
  bool apart = false; // two problems that are launched one after the other (nothing else is set then)
  bool on_host() const { return split > 0 || apart; }      // nothing has been uploaded
  int cg = 1;         // CTAs per tile
  int grid = 0;       // workers (CTAs, or pairs of CTAs)
  int* d_offsets = nullptr;
  int* d_items = nullptr;
  unsigned long long last_use = 0;
};
// Cache of uploaded schedules, keyed by (device, M, N, K, epilogue of every problem).  A training run uses a
// few dozen shape sets; callers whose row counts change from call to call (expert-parallel MoE)
// use the ragged kernel instead, which takes the counts from device memory and needs no schedule.
// The cache is still bounded: beyond MAX_SCHEDULES entries the least recently used one is freed.  Entries of the split form are only a number
// on the host: they have a limit of their own and push out no uploaded schedule, which takes allocations and synchronous copies to make again.
constexpr int MAX_SCHEDULES = 128, MAX_SPLITS = 512;
std::map<std::vector<int>, Schedule> g_schedules;
int g_cached[2] = {0, 0};      // entries with a schedule, entries of the split form
unsigned long long g_sched_clock = 0;
std::mutex g_sched_mutex;
int g_sms = 0;

// Longest tiles first, each to the least loaded CTA (ties: lowest CTA index, which keeps tiles
// that run at the same time adjacent in the problem's L2-friendly order).
struct Item { int cost, code; };

// Modelled time of a tile, in hundredths of a single CTA's k-block: the main loop plus a fixed part, but not less than storing
// the tile takes.  A pair's k-block takes less of the tensor pipe, its two stores run in step and hide less.
long long tile_time(int num_kb, int cg) {
  return cg == 1 ? std::max(100LL * num_kb + 800, 1200LL) : std::max(86LL * num_kb + 800, 25LL * num_kb + 1700);
}

// The assignment itself (host only): per-worker item lists, longest tiles first, each to the least
// loaded worker.  Returns the load (in k-block units) of the busiest one; `time` receives its modelled time.
long long assign_items(const Problem* probs, int np, int cg, int sms, std::vector<std::vector<int>>* per_out, int* total_out,
                       long long* work_out, long long* time_out) {
  std::vector<Item> items;
  std::vector<int> order(np);
  for (int i = 0; i < np; i++) order[i] = i;
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return probs[a].num_kb > probs[b].num_kb; });
  long long work = 0;
  for (int oi = 0; oi < np; oi++) {
    const int i = order[oi];
    const int nt = probs[i].tiles_m * probs[i].tiles_n;
    if (nt >= (1 << 24)) return -1;
    for (int t = 0; t < nt; t++) {
      items.push_back({probs[i].num_kb + 6, (i << 24) | t});   // +6: fixed cost per tile
      work += probs[i].num_kb + 6;
    }
  }
  const int total = (int)items.size();
  const int workers = sms / cg;
  const int grid = total < workers ? total : workers;
  typedef std::pair<long long, int> Load;
  std::priority_queue<Load, std::vector<Load>, std::greater<Load>> heap;
  for (int c = 0; c < grid; c++) heap.push({0, c});
  std::vector<std::vector<int>> per(grid);
  std::vector<long long> time(grid, 0);
  long long busiest = 0;
  for (const Item& it : items) {
    Load l = heap.top();
    heap.pop();
    per[l.second].push_back(it.code);
    time[l.second] += tile_time(it.cost - 6, cg);
    const long long load = l.first + it.cost;
    if (load > busiest) busiest = load;
    heap.push({load, l.second});
  }
  if (per_out) per_out->swap(per);
  if (total_out) *total_out = total;
  if (work_out) *work_out = work;
  if (time_out) *time_out = *std::max_element(time.begin(), time.end());
  return busiest;
}

void set_tiles(Problem* p, int cg) {
  p->tiles_m = (p->M + BM * cg - 1) / (BM * cg);
  p->tiles_n = (p->N + BN - 1) / BN;
  p->num_kb = (p->K + BK - 1) / BK;
}

// CTAs per tile for this set of problems: the form whose busiest worker is modelled to finish first (tile_time, plus 6 k-blocks for
// setting up the pairs of a launch).  Fitted to 727 launches in both forms: 130 to 16384 rows, N 768 to 11264, K 128 to 8192, all
// operand majors, data + weight gradients, SwiGLU epilogues; the rule is on average 0.1 % off the better form, and at worst 6 % (launches
// of one tile per CTA).  CTAs / pairs in us: where the store of a tile outlasts its main loop, 16384 x 4096 x 256 64.6 / 79.8,
// x 512 80.0 / 88.9, 8192 x 4096 x 768 51.2 / 52.4; where it does not, 8192 x 4096 x 1024 62.1 / 58.7, 16384 x 4096 x 1536 167 / 150,
// 4096 x 11264 x 4096 287 / 259; short launches, 1000 x 2304 x 768 14.6 / 16.5, 1000 x 768 x 4096 31.2 / 30.3.
int choose_cg(Problem* probs, int np, int sms, long long* best = nullptr) {
  if (sms < 2) return 1;
  long long time[3] = {0, 0, 0};
  for (int cg = 1; cg <= 2; cg++) {
    for (int i = 0; i < np; i++) set_tiles(&probs[i], cg);
    if (assign_items(probs, np, cg, sms, nullptr, nullptr, nullptr, &time[cg]) < 0) return -1;
  }
  const int cg = time[2] + 600 < time[1] ? 2 : 1;
  if (best) *best = cg == 2 ? time[2] + 600 : time[1];
  return cg;
}

int parts_of(const Problem* probs, int np, int sms, long long list_time, double* us = nullptr) {
  int M[MAX_PROBLEMS], N[MAX_PROBLEMS], K[MAX_PROBLEMS];
  bool activation = false;
  for (int i = 0; i < np; i++) {
    M[i] = probs[i].M; N[i] = probs[i].N; K[i] = probs[i].K;
    activation |= probs[i].epi == 1 || probs[i].epi == 2;
  }
  return gemm_split_parts(np, M, N, K, activation, sms, list_time, us);
}

// Whether two problems are better launched one after the other: a weight gradient over few rows is many short tiles, its data gradient a few tiles with a
// long reduction, each of which a list gives to one worker.  On its own the latter is split.  Alone, short tiles take the time of their bytes (5.3 TB/s) and of
// their waves; 5 us are kept back for the second launch.  Together / apart, us (n x k weights, T rows): 32000 x 768, T 64 149 / 42; 11264 x 2048, T 64 59 / 29, T
// 256 60 / 40; 28672 x 4096, T 16 182 / 100; 8192 x 1024, T 496 44 / 30; 4096 x 768, T 64 25 / 20.  Passes of launches below 40 us are bound by the host (a
// feed-forward of 64 x 768 takes 85 us of it and 47 of the GPU), to which a second launch only adds.
bool better_apart(const Problem* probs, int np, int sms, long long list_time, double joint_us) {
  if (np != 2 || sms < 4 || joint_us < 40.0) return false;
  const int longest = std::max((probs[0].K + BK - 1) / BK, (probs[1].K + BK - 1) / BK);
  if (100.0 * longest + 800 < 0.6 * (double)list_time) return false;
  double alone = -2.0;
  for (int i = 0; i < 2; i++) {
    Problem p = probs[i];
    long long time = 0;
    double us = 0;
    if (choose_cg(&p, 1, sms, &time) < 0) return false;
    parts_of(&p, 1, sms, time, &us);
    set_tiles(&p, 1);
    const double mb = 2e-6 * ((double)p.M * p.K + (double)p.N * p.K + (double)p.M * p.N);
    const double waves = std::ceil((double)p.tiles_m * p.tiles_n / sms);
    alone += std::min(us, 5.0 + 0.19 * mb + 0.27 * waves * p.num_kb);
  }
  return alone + 5.0 < 0.93 * joint_us;
}

int build_schedule(Problem* probs, int np, int sms, Schedule* out) {
  std::vector<std::vector<int>> per;
  int total = 0;
  long long time = 0;
  out->cg = choose_cg(probs, np, sms, &time);
  if (out->cg < 0) return LB_ERR_SHAPE;
  double us = 0;
  if (time > 0) out->split = parts_of(probs, np, sms, time, &us);
  if (time > 0 && better_apart(probs, np, sms, time, us)) { out->split = 0; out->apart = true; }
  if (out->on_host()) return LB_OK;
  for (int i = 0; i < np; i++) set_tiles(&probs[i], out->cg);
  if (assign_items(probs, np, out->cg, sms, &per, &total, nullptr, nullptr) < 0) return LB_ERR_SHAPE;
  const int grid = (int)per.size();
  std::vector<int> offsets(grid + 1, 0), flat;
  flat.reserve(total);
  for (int c = 0; c < grid; c++) {
    offsets[c] = (int)flat.size();
    flat.insert(flat.end(), per[c].begin(), per[c].end());
  }
  offsets[grid] = (int)flat.size();
  if (cudaMalloc(&out->d_offsets, sizeof(int) * (grid + 1)) != cudaSuccess) return LB_ERR_LAUNCH;
  if (cudaMalloc(&out->d_items, sizeof(int) * (total > 0 ? total : 1)) != cudaSuccess) return LB_ERR_LAUNCH;
  cudaMemcpy(out->d_offsets, offsets.data(), sizeof(int) * (grid + 1), cudaMemcpyHostToDevice);
  cudaMemcpy(out->d_items, flat.data(), sizeof(int) * total, cudaMemcpyHostToDevice);
  out->grid = grid;
  return LB_OK;
}

// Map of the boxes of 32 rows that an epilogue warp stores.
int out_map(CUtensorMap* m, const bf16* base, int cols, int rows, long long ld) {
  return bw::make_map_bf16(m, base, (uint64_t)cols, (uint64_t)rows, (uint64_t)ld, 64, 32);
}
// The maps of a problem's outputs (see GroupedParams::tc).
int out_maps(CUtensorMap* tc, void* C, void* C2, long long ldc, long long ldc2, int rows, int N, int epi, int half) {
  bf16* c = (bf16*)C;
  if (epi == 2) return LB_OK;
  if (epi != 1) return out_map(tc, c, N, rows, ldc);
  int rc = c ? out_map(tc, c, half, rows, ldc) : LB_OK;
  if (!rc && c) rc = out_map(tc + 1, c + half, half, rows, ldc);
  return rc ? rc : out_map(tc + 2, (const bf16*)C2, half, rows, ldc2);
}

// Launches a form of a kernel on `workers` workers; a pair is a cluster of two CTAs.
template <typename C, typename P>
int launch_form(void (*fn)(P), C, int cg, int workers, bool dependent, const P& params, cudaStream_t s) {
  {
    std::lock_guard<std::mutex> lock(g_sched_mutex);
    static std::vector<const void*> ready;      // (of this configuration)
    const void* f = reinterpret_cast<const void*>(fn);
    if (std::find(ready.begin(), ready.end(), f) == ready.end()) {
      if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES) != cudaSuccess) return LB_ERR_LAUNCH;
      ready.push_back(f);
    }
  }
  return lb_launch_cluster(dependent, cg, fn, cg * workers, C::NUM_THREADS, C::SMEM_BYTES, s, params);
}

struct Operands {
  const void *const *A, *const *B;
  void *const *C, *const *C2;
  const long long *lda, *ldb, *ldc, *ldc2;
  const RopeArgs* rope;
};
template <int NP>
int launch_grouped(int n, const Problem* probs, const Operands& op, const Schedule& sched, cudaStream_t s) {
  static thread_local GroupedParams<NP> gp;         // up to 5.5 KB of tensor maps: kept off the stack, one per calling thread
  for (int i = 0; i < n; i++) {
    const Problem& p = gp.prob[i] = probs[i];
    int rc;
    if (!p.a_mn) rc = bw::make_map_bf16(&gp.ta[i], op.A[i], (uint64_t)p.K, (uint64_t)p.M, (uint64_t)op.lda[i], BK, BM);
    else         rc = bw::make_map_bf16(&gp.ta[i], op.A[i], (uint64_t)p.M, (uint64_t)p.K, (uint64_t)op.lda[i], 64, BK);
    if (rc) return rc;
    if (!p.b_mn) rc = bw::make_map_bf16(&gp.tb[i], op.B[i], (uint64_t)p.K, (uint64_t)p.N, (uint64_t)op.ldb[i], BK, BN / 2);
    else         rc = bw::make_map_bf16(&gp.tb[i], op.B[i], (uint64_t)p.N, (uint64_t)p.K, (uint64_t)op.ldb[i], 64, BK);
    if (rc) return rc;
    if ((rc = out_maps(gp.tc[i], op.C[i], op.C2 ? op.C2[i] : nullptr, op.ldc[i], op.ldc2 ? op.ldc2[i] : 0, p.M, p.N, p.epi, p.half))) return rc;
  }
  gp.rope = op.rope ? *op.rope : RopeArgs{nullptr, nullptr, nullptr, 1, 64, 0};
  gp.offsets = sched.d_offsets;
  gp.items = sched.d_items;
  const bool eight = std::any_of(probs, probs + n, [](const Problem& p) { return p.epi == 2; });
  if (sched.cg == 2) return eight ? launch_form(gemm_grouped_kernel<2, 8, NP>, Cfg<2, 8>(), 2, sched.grid, true, gp, s)
                                  : launch_form(gemm_grouped_kernel<2, 4, NP>, Cfg<2, 4>(), 2, sched.grid, true, gp, s);
  return eight ? launch_form(gemm_grouped_kernel<1, 8, NP>, Cfg<1, 8>(), 1, sched.grid, true, gp, s)
               : launch_form(gemm_grouped_kernel<1, 4, NP>, Cfg<1, 4>(), 1, sched.grid, true, gp, s);
}

}  // namespace

// Copies the status words of the grouped GEMM kernel to host memory and clears them.
extern "C" int lb_gemm_grouped_status(void* out) {
  cudaError_t e = cudaMemcpyFromSymbol(out, g_grp_status, sizeof(unsigned int) * 4);
  if (e != cudaSuccess) { g_lb_last_cuda_error = (int)e; return LB_ERR_LAUNCH; }
  unsigned int zeros[4] = {0, 0, 0, 0};
  cudaMemcpyToSymbol(g_grp_status, zeros, sizeof(zeros));
  return LB_OK;
}

// Number of schedules currently cached (never more than MAX_SCHEDULES).
extern "C" int lb_gemm_grouped_cached() {
  std::lock_guard<std::mutex> lock(g_sched_mutex);
  return g_cached[0];
}

namespace {
// Problems of the host-only entry points below; false for sizes that no launch takes.
bool plan_problems(int n, const int* M, const int* N, const int* K, int sms, Problem* probs) {
  if (n < 1 || n > MAX_PROBLEMS || sms < 1) return false;
  for (int i = 0; i < n; i++) {
    if (M[i] <= 0 || N[i] <= 0 || K[i] <= 0) return false;
    probs[i].M = M[i]; probs[i].N = N[i]; probs[i].K = K[i];
    probs[i].epi = 0;
  }
  return true;
}
}  // namespace

// Host only (no CUDA call): parts of K (1, 2, 4 or 8) with which lb_gemm_grouped gives these shapes to the split form (gemm_split.cu), 0 where
// it takes the list form, which the two entry points below describe.
extern "C" int lb_gemm_grouped_parts(int n, const int* M, const int* N, const int* K, int sms) {
  Problem probs[MAX_PROBLEMS];
  if (!plan_problems(n, M, N, K, sms, probs)) return LB_ERR_SHAPE;
  long long time = 0;
  if (choose_cg(probs, n, sms, &time) < 0) return LB_ERR_SHAPE;
  return time > 0 ? parts_of(probs, n, sms, time) : 0;
}

// Host only (no CUDA call): 1 where lb_gemm_grouped launches two plain problems one after the other instead of together.
extern "C" int lb_gemm_grouped_apart(int n, const int* M, const int* N, const int* K, int sms) {
  Problem probs[MAX_PROBLEMS];
  if (!plan_problems(n, M, N, K, sms, probs)) return LB_ERR_SHAPE;
  long long time = 0;
  double us = 0;
  if (choose_cg(probs, n, sms, &time) < 0) return LB_ERR_SHAPE;
  if (time > 0) parts_of(probs, n, sms, time, &us);
  return time > 0 && better_apart(probs, n, sms, time, us);
}

// Host only (no CUDA call): CTAs per tile, 1 or 2, of the schedule that lb_gemm_grouped builds for these shapes on `sms` SMs.
extern "C" int lb_gemm_grouped_ctas_per_tile(int n, const int* M, const int* N, const int* K, int sms) {
  Problem probs[MAX_PROBLEMS];
  if (!plan_problems(n, M, N, K, sms, probs)) return LB_ERR_SHAPE;
  const int cg = choose_cg(probs, n, sms);
  return cg < 0 ? LB_ERR_SHAPE : cg;
}

// Host only (no CUDA call): that schedule.  out[0] = load of the busiest CTA, out[1] = total work, out[2] = number of CTAs used,
// all in k-block units of 64 (a tile counts its k-blocks + 6, for each of its CTAs).  busiest * CTAs / total is the imbalance factor.
extern "C" int lb_gemm_grouped_plan(int n, const int* M, const int* N, const int* K, int sms, long long* out) {
  Problem probs[MAX_PROBLEMS];
  if (!plan_problems(n, M, N, K, sms, probs)) return LB_ERR_SHAPE;
  const int cg = choose_cg(probs, n, sms);
  if (cg < 0) return LB_ERR_SHAPE;
  for (int i = 0; i < n; i++) set_tiles(&probs[i], cg);
  std::vector<std::vector<int>> per;
  int total = 0;
  long long work = 0;
  const long long busiest = assign_items(probs, n, cg, sms, &per, &total, &work, nullptr);
  if (busiest < 0) return LB_ERR_SHAPE;
  out[0] = busiest; out[1] = cg * work; out[2] = cg * (long long)per.size();
  return LB_OK;
}

// n problems (1..8), arrays of length n.  Per problem the rules of lb_gemm_bf16 apply: pointers
// 16-byte aligned, lda / ldb / ldc / N multiples of 8 (M too when a_mn).  accumulate[i] != 0 adds
// the product to the old contents of C_i.  The first call with a new set of shapes builds and
// uploads the schedule (two small device allocations, synchronous copies); later calls only launch.  Launches of one or two problems that
// do not fill the chip go to the split form (gemm_split.cu), which has no schedule to upload.
//
// lb_gemm_grouped_epi additionally takes, per problem, an epilogue selector (see `Problem`), a second
// matrix C2 with its leading dimension, and `half`:
//   epi 1: B is a fused [2 * half, K] gate | up weight (b_mn = 0), N = 2 * half, C [M, 2 * half] receives
//          g | u (nothing, with a null C) and C2 [M, half] receives silu(g) * u;
//   epi 2: N = half, the product is dh; C2 [M, 2 * half] holds g | u and C [M, 2 * half] receives dg | du.
static int run_grouped(int n, const void* const* A, const void* const* B, void* const* C, const int* M, const int* N, const int* K,
                       const long long* lda, const long long* ldb, const long long* ldc, const int* a_mn, const int* b_mn, const int* accumulate,
                       const int* epi, void* const* C2, const long long* ldc2, const int* half, const RopeArgs* rope, void* stream) {
  if (n < 1 || n > MAX_PROBLEMS) return LB_ERR_SHAPE;
  Problem probs[MAX_PROBLEMS];
  std::vector<int> key;
  int dev = 0;
  cudaGetDevice(&dev);
  key.push_back(dev);
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
    }
    Problem& p = probs[i];
    p.M = M[i]; p.N = N[i]; p.K = K[i]; p.epi = rope ? 4 : e; p.half = e ? half[i] : 0; p.keep = C[i] != nullptr;
    p.old = (const bf16*)(e == 2 ? C2[i] : C[i]); p.ld_old = e == 2 ? ldc2[i] : ldc[i]; p.C = (bf16*)C[i]; p.ldc = ldc[i];
    p.a_mn = a_mn[i]; p.b_mn = b_mn[i]; p.accumulate = accumulate ? accumulate[i] : 0;
    key.push_back(M[i]); key.push_back(N[i]); key.push_back(K[i]); key.push_back(e);
  }
  {
    std::lock_guard<std::mutex> lock(g_sched_mutex);
    if (g_sms == 0 && cudaDeviceGetAttribute(&g_sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
      cudaGetLastError();
      g_sms = 0;
      return LB_ERR_LAUNCH;
    }
  }
  Schedule sched;
  {
    std::lock_guard<std::mutex> lock(g_sched_mutex);
    auto it = g_schedules.find(key);
    if (it == g_schedules.end()) {
      Schedule s;
      int rc = build_schedule(probs, n, g_sms, &s);
      if (rc) return rc;
      const bool split = s.on_host();
      if (++g_cached[split] > (split ? MAX_SPLITS : MAX_SCHEDULES)) {
        // evict the least recently used entry of its kind; cudaFree waits for kernels that may still read it
        auto victim = g_schedules.end();
        for (auto j = g_schedules.begin(); j != g_schedules.end(); ++j)
          if (j->second.on_host() == split && (victim == g_schedules.end() || j->second.last_use < victim->second.last_use)) victim = j;
        if (!split) {
          cudaFree(victim->second.d_offsets);
          cudaFree(victim->second.d_items);
        }
        g_schedules.erase(victim);
        g_cached[split]--;
      }
      it = g_schedules.emplace(key, s).first;
    }
    it->second.last_use = ++g_sched_clock;
    sched = it->second;
  }
  if (sched.apart) {
    for (int i = 0; i < n; i++) {
      const int rc = run_grouped(1, A + i, B + i, C + i, M + i, N + i, K + i, lda + i, ldb + i, ldc + i, a_mn + i, b_mn + i, accumulate ? accumulate + i : nullptr,
                                 epi ? epi + i : nullptr, C2 ? C2 + i : nullptr, ldc2 ? ldc2 + i : nullptr, half ? half + i : nullptr, nullptr, stream);
      if (rc) return rc;
    }
    return LB_OK;
  }
  if (sched.split)
    return gemm_split_rope(n, A, B, C, M, N, K, lda, ldb, ldc, a_mn, b_mn, accumulate, epi, C2, ldc2, half, sched.split, rope, stream);
  for (int i = 0; i < n; i++) set_tiles(&probs[i], sched.cg);
  const Operands op{A, B, C, epi ? C2 : nullptr, lda, ldb, ldc, epi ? ldc2 : nullptr, rope};
  return n <= 2 ? launch_grouped<2>(n, probs, op, sched, (cudaStream_t)stream) : launch_grouped<MAX_PROBLEMS>(n, probs, op, sched, (cudaStream_t)stream);
}


extern "C" int lb_gemm_grouped_epi(int n, const void* const* A, const void* const* B, void* const* C, const int* M,
                                   const int* N, const int* K, const long long* lda, const long long* ldb,
                                   const long long* ldc, const int* a_mn, const int* b_mn, const int* accumulate,
                                   const int* epi, void* const* C2, const long long* ldc2, const int* half,
                                   void* stream) {
  return run_grouped(n, A, B, C, M, N, K, lda, ldb, ldc, a_mn, b_mn, accumulate, epi, C2, ldc2, half, nullptr, stream);
}

// C [M, N] = X [M, K] W^T (W [N, K]; all matrices contiguous) with the first rope_cols columns, heads of head_dim columns, rotated as
// lb_rope rotates them: row r is token r of sequences of S tokens.
extern "C" int lb_gemm_rope(const void* X, const void* W, void* C, int M, int N, int K, const void* cosT, const void* sinT, const void* positions,
                            int S, int head_dim, int rope_cols, void* stream) {
  if (S <= 0 || head_dim <= 0 || (head_dim % 8) || rope_cols < 0 || rope_cols > N || (rope_cols % head_dim)) return LB_ERR_SHAPE;
  const RopeArgs rope{(const float*)cosT, (const float*)sinT, (const int*)positions, S, head_dim, rope_cols};
  const long long lda = K, ldb = K, ldc = N;
  const int k_major = 0;
  return run_grouped(1, &X, &W, &C, &M, &N, &K, &lda, &ldb, &ldc, &k_major, &k_major, nullptr, nullptr, nullptr, nullptr, nullptr, &rope, stream);
}

extern "C" int lb_gemm_grouped(int n, const void* const* A, const void* const* B, void* const* C, const int* M,
                               const int* N, const int* K, const long long* lda, const long long* ldb,
                               const long long* ldc, const int* a_mn, const int* b_mn, const int* accumulate,
                               void* stream) {
  return lb_gemm_grouped_epi(n, A, B, C, M, N, K, lda, ldb, ldc, a_mn, b_mn, accumulate, nullptr, nullptr, nullptr, nullptr,
                             stream);
}

namespace {
// CTAs per tile.  The rows are known on the device only: as many as the caller expects in all, the same for every expert, half a tile of each
// wasted.  (Not as many as the buffer holds: between several GPUs its capacity is twice what arrives on average.)  Both forms' times as tile_time() has them for the lists (a pair's as those of a launch, 6 k-blocks more), 3 % for the
// unevenness, which costs pairs more.  CTAs / pairs in us, 8 experts, 2048 -> 4096, 2 of them per token, 4096 tokens: gate | up 254 / 220, down 127 / 106, its data
// gradient 143 / 144, gate | up's 251 / 252; 1024 tokens 88 / 77, 60 / 54, 64 / 60, 107 / 96; 64 tokens 54 / 63, 34 / 33, 38 / 44, 56 / 58; 4096 tokens of 4
// experts, 1024 -> 4096: 131 / 108, 59 / 55, 124 / 127, 111 / 104.
int ragged_cg(int LE, int all_rows, int n, int num_kb, int sms) {
  if (sms < 2) return 1;
  const double rows = std::max(1.0, (double)all_rows / LE);
  const double tn = (n + BN - 1) / BN;
  double time[3];
  for (int cg = 1; cg <= 2; cg++) {
    const double tiles = LE * std::max(1.0, rows / (BM * cg) + 0.5) * tn;
    time[cg] = std::ceil(tiles / (sms / cg)) * (double)tile_time(num_kb, cg);
  }
  return 1.03 * (time[2] + 600) < time[1] ? 2 : 1;
}
// Weight gradients: as many tiles whatever the rows are, but with few of them a tile is mostly its store.  CTAs / pairs, down and gate | up: 1024 rows per expert
// 126 / 118 and 282 / 222, 512 90 / 79 and 158 / 137, 256 48 / 59 and 88 / 105.  (Uneven routing, 8 experts, 512 rows on average 72 / 67 and 135 / 126, 448 65 / 62 and 122 /
// 116, 384 60 / 59 and 110 / 109, 256 47 / 57 and 86 / 103.)
int ragged_wgrad_cg(int LE, int all_rows, int sms) {
  return sms >= 2 && all_rows / LE >= 512 ? 2 : 1;
}
// Rows to expect: the caller's number, or, where that is 0, what the buffer holds beyond the padding of its segments.
int ragged_rows(int LE, int cap, int rows) { return rows > 0 ? rows : cap - LE * BM; }
int launch_ragged(int cg, bool dependent, const RaggedParams& rp, cudaStream_t s) {
  const int workers = lb_num_sms() / cg;
  if (cg == 2) return rp.epi == 2 ? launch_form(gemm_ragged_kernel<2, 8>, Cfg<2, 8>(), 2, workers, dependent, rp, s)
                                  : launch_form(gemm_ragged_kernel<2, 4>, Cfg<2, 4>(), 2, workers, dependent, rp, s);
  return rp.epi == 2 ? launch_form(gemm_ragged_kernel<1, 8>, Cfg<1, 8>(), 1, workers, dependent, rp, s)
                     : launch_form(gemm_ragged_kernel<1, 4>, Cfg<1, 4>(), 1, workers, dependent, rp, s);
}
}  // namespace

// Host only (no CUDA call): CTAs per tile, 1 or 2, of an expert GEMM over a buffer of `cap` rows (K > 0) of which as many are expected as it holds, or of its weight
// gradient (K = 0), on `sms` SMs.
extern "C" int lb_gemm_ragged_ctas_per_tile(int LE, int cap, int N, int K, int sms) {
  if (LE < 1 || LE > MAX_PROBLEMS || cap <= 0 || N <= 0 || K < 0 || sms < 1) return LB_ERR_SHAPE;
  const int rows = ragged_rows(LE, cap, 0);
  return K ? ragged_cg(LE, rows, N, (K + BK - 1) / BK, sms) : ragged_wgrad_cg(LE, rows, sms);
}

// Expert GEMMs over ragged row segments (see gemm_ragged_kernel).  seg: device table of 2 * LE + 2
// ints (offsets, counts, ...), LE <= 8 local experts.
//  mode 0: C [cap, N] = A [cap, K] . op(B_e)^T per segment; B: host array of LE weight pointers
//          ([N, K], or [K, N] with b_mn), all with leading dimension ldb.  wait_flag (or null): device
//          word that must reach wait_target before A is read.
//          epi, C2, ldc2 and half as in lb_gemm_grouped_epi (matrices of cap rows).
//  rows: how many there will be in all segments, as far as the caller can tell, or 0 (as many as fit); it decides which form runs, not what is computed.
extern "C" int lb_gemm_ragged_epi(const void* A, const void* const* B, void* C, const void* seg, int LE, int cap, int rows, int N, int K,
                                  long long lda, long long ldb, long long ldc, int b_mn, int epi, void* C2, long long ldc2, int half,
                                  const void* wait_flag, unsigned int wait_target, void* stream) {
  if (LE < 1 || LE > MAX_PROBLEMS || cap <= 0 || N <= 0 || K <= 0) return LB_ERR_SHAPE;
  if ((lda % 8) || (ldb % 8) || (ldc % 8) || (N % 8) || (K % 8)) return LB_ERR_SHAPE;
  if (((uintptr_t)A | (uintptr_t)C) & 15) return LB_ERR_ARG;
  if (epi < 0 || epi > 2 || (!C && epi != 1)) return LB_ERR_ARG;
  if (epi) {
    if (!C2 || ((uintptr_t)C2 & 15) || (ldc2 % 8) || half <= 0 || (half % 8)) return LB_ERR_ARG;
    if (epi == 1 ? (b_mn || N != 2 * half) : N != half) return LB_ERR_SHAPE;
  }
  static thread_local RaggedParams rp;
  int rc = bw::make_map_bf16(&rp.ta, A, (uint64_t)K, (uint64_t)cap, (uint64_t)lda, BK, BM);
  if (rc) return rc;
  for (int e = 0; e < LE; e++) {
    if ((uintptr_t)B[e] & 15) return LB_ERR_ARG;
    if (!b_mn) rc = bw::make_map_bf16(&rp.tb[e], B[e], (uint64_t)K, (uint64_t)N, (uint64_t)ldb, BK, BN / 2);
    else       rc = bw::make_map_bf16(&rp.tb[e], B[e], (uint64_t)N, (uint64_t)K, (uint64_t)ldb, 64, BK);
    if (rc) return rc;
    rp.C[e] = nullptr;
  }
  if ((rc = out_maps(rp.tc, C, C2, ldc, ldc2, cap, N, epi, half))) return rc;
  rp.C[0] = (bf16*)C; rp.ldc = ldc; rp.old = (const bf16*)C2; rp.ld_old = ldc2; rp.epi = epi; rp.half = half; rp.keep = C != nullptr; rp.seg = (const int*)seg; rp.LE = LE; rp.M_w = 0; rp.N = N; rp.K = K; rp.b_mn = b_mn;
  rp.mode = 0; rp.accumulate = 0; rp.cap = cap;
  rp.tiles_n = (N + BN - 1) / BN; rp.tiles_m_w = 0; rp.num_kb = (K + BK - 1) / BK;
  rp.wait_flag = (const unsigned int*)wait_flag; rp.wait_target = wait_target; rp.wait_ns = g_lb_flag_wait_ns;
  return launch_ragged(ragged_cg(LE, ragged_rows(LE, cap, rows), N, rp.num_kb, lb_num_sms()), !wait_flag, rp, (cudaStream_t)stream);
}

//  Weight gradients: C_e [Nw, Kw] (+)= dY[rows of e, Nw]^T . X[rows of e, Kw]; C: host array of LE
//  gradient pointers with leading dimension ldc.  Without accumulate every C_e is written whole (zeros for an expert
//  without rows).
extern "C" int lb_gemm_ragged_wgrad(const void* dY, const void* X, void* const* C, const void* seg, int LE, int cap, int rows, int Nw,
                                    int Kw, long long lddy, long long ldx, long long ldc, int accumulate, void* stream) {
  if (LE < 1 || LE > MAX_PROBLEMS || cap <= 0 || Nw <= 0 || Kw <= 0) return LB_ERR_SHAPE;
  if ((lddy % 8) || (ldx % 8) || (ldc % 8) || (Nw % 8) || (Kw % 8)) return LB_ERR_SHAPE;
  if (((uintptr_t)dY | (uintptr_t)X) & 15) return LB_ERR_ARG;
  for (int e = 0; e < LE; e++)
    if (!C[e] || ((uintptr_t)C[e] & 15)) return LB_ERR_ARG;
  static thread_local RaggedParams rp;
  const int cg = ragged_wgrad_cg(LE, ragged_rows(LE, cap, rows), lb_num_sms());
  int rc = bw::make_map_bf16(&rp.ta, dY, (uint64_t)Nw, (uint64_t)cap, (uint64_t)lddy, 64, BK);
  if (rc) return rc;
  rc = bw::make_map_bf16(&rp.tb[0], X, (uint64_t)Kw, (uint64_t)cap, (uint64_t)ldx, 64, BK);
  if (rc) return rc;
  for (int e = 0; e < LE; e++) {
    rp.C[e] = (bf16*)C[e];
    if ((rc = out_map(&rp.tc[e], rp.C[e], Kw, Nw, ldc))) return rc;
  }
  rp.ldc = ldc; rp.old = nullptr; rp.ld_old = 0; rp.epi = 0; rp.half = 0; rp.keep = 1; rp.seg = (const int*)seg; rp.LE = LE; rp.M_w = Nw; rp.N = Kw; rp.K = 0; rp.b_mn = 1; rp.mode = 1;
  rp.accumulate = accumulate; rp.cap = cap;
  rp.tiles_n = (Kw + BN - 1) / BN; rp.tiles_m_w = (Nw + BM * cg - 1) / (BM * cg); rp.num_kb = 0;
  rp.wait_flag = nullptr; rp.wait_target = 0; rp.wait_ns = g_lb_flag_wait_ns;
  return launch_ragged(cg, true, rp, (cudaStream_t)stream);
}
