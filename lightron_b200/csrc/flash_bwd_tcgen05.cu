// FlashAttention backward on the 5th-generation tensor cores (sm_100a), head_dim 64 or 128.
//
// One CTA owns a block of 128 keys of one (batch, kv head) and walks over every 128-query block
// (of every query head of the GQA group) that can see it.  Scores are computed TRANSPOSED, keys in the rows:
//     S^T  = K Q^T           [128 k x 128 q]   (K-major operands in shared memory)
//     dP^T = V dO^T          [128 k x 128 q]
//     dV  += P^T dO          [128 k x d]       A = P^T from tensor memory, B = dO MN-major
//     dK  += dS^T Q          [128 k x d]       A = dS^T from tensor memory, B = Q MN-major
//     dQ   = dS K            [128 q x d]       A = dS as MN-major operand, B = K MN-major
// A thread of the math warps owns a key row (and 64 of the 128 queries): P^T and dS^T go back to tensor memory as
// packed bf16, where they are the A operands of dV and dK as they lie.  Only dS is also written to shared memory, once,
// for dQ.  With the query rows in the lanes (the form this replaced) P and dS both passed through shared
// memory and every math, gradient and drain phase of a block waited for the one before it.
// S^T, dP^T, dV, dK live in TMEM (dV / dK accumulate there across the whole loop, so no rescaling is ever
// needed); P^T takes columns of S^T, dS^T columns of dP^T, and with head_dim 128 (512 columns full) dQ takes
// those of dP^T.  The tensor pipe runs MMAs in issue order, so a region is reused without a wait when both uses are MMAs:
//     dV(i) | S(i+1) | dK(i) | dQ(i) | dP(i+1)      (head_dim 64: dP(i+1) before dQ(i))
// The exponentials of block i+1 therefore run under dK / dQ of block i.  Each dQ tile is drained by four warps of
// their own: TMEM -> registers (a whole row, so that the columns are free at once) -> staging -> asynchronous bulk reduce-add
// (cp.reduce.async.bulk .add.f32) into an fp32 accumulator in global memory, whose layout is the staging layout (un-permuted by the final
// convert kernel), so no atomic instructions pass through the load/store pipe (16-byte reductions straight from the registers held
// up every other access of the SM: 5360 against 3750 cycles a block at d = 128).
// What bounds it.  Cycles of a block: d = 64 2770, of which the math warps are never idle (exponentials 1330, dS 480, the rest waits, stores
// and tensor-memory accesses); d = 128 3750, the chain dS -> dK, dQ -> drain -> dP of the next block, which shares dQ's columns, against 2560 of
// tensor pipe.  Both run at the power limit in long loops (1.64 / 1.53 GHz).  Counters: tensor pipe 45 / 58 %, L1 and shared memory 55 / 73 %,
// exponentials 36 / 23 % of the active cycles (B8 S2048 32q/4kv d64, B4 S2048 32q/8kv d128).  What it took to get there from 3150 / 4500: an elected thread
// that issues (elect_one), one arrival per warp, waits that are sure to succeed ahead of the one that is not, no divisions in the loops,
// dQ's columns freed after 110 instead of 800 cycles, dK and dV through TMA stores (prologue and stores of a CTA: 12000 / 16000 cycles before).
// Loops of 0.35 s of all its kernels, before / now, on one GPU: B8 S2048 32q/4kv d64 646 / 547 us, B1 S8192 32q/8kv d128
// 1624 / 1404, B3 S1531 32q/8kv d128 237 / 221, B1 S4096 8q/8kv d128 117 / 104.
// A key block's loop over query blocks may be cut into parts of `chunk` blocks, a CTA each, where whole loops would leave SMs without work (a causal
// sequence's first key block takes as long as all blocks of the last ones together, and grouped heads make few CTAs of long loops): each part then leaves its
// dK / dV in fp32 in a place of its own, and the kernel that converts dQ adds them up, in the order of the parts: dK and dV are the same bits in every run, as
// those of whole loops are (dQ, to which the key blocks add as they come, is not, beyond 128 keys).  bwd_chunk() has the rule and the figures.
// Warp roles (512 threads): warp 0 TMA producer, warp 1 MMA issuer + TMEM owner, warps 4-11 math, 12-15 dQ drain.
// All waits are bounded; on expiry a status word is set and the CTA drains and frees its TMEM.
#include <algorithm>
#include "tcgen05.cuh"

static __device__ unsigned int g_fab_status[4] = {0, 0, 0, 0};

namespace {
using namespace bw;

struct FaBwdParams {
  const bf16 *o, *dout;
  const float* lse;
  float *stats, *dq_acc;
  bf16 *dq, *dk, *dv;
  int B, Sq, Sk, hq, hkv;
  long long o_ts, do_ts, dq_ts, dk_ts, dv_ts;
  float scale;
  int causal;
  int kv_brows;   // rows between consecutive batches in the K/V tensor maps (>= Sk)
  int chunk;      // query blocks of a CTA, or 0: all of its key block, whose dK / dV it writes
  float *dk_acc, *dv_acc;      // with chunk: a tile in the layout of dq_acc's for every CTA of the launch
  bool alone;                  // one key block, not in parts: its CTAs write dQ, and nothing uses dq_acc
};

// (batch, kv head) pairs whose key blocks are ordered together: enough to keep the chip busy to the end,
// few enough that several key blocks of a pair run at a time and share its Q / dO / dQ traffic in L2.
constexpr int BWD_GROUP = 32;

template <int D>
struct BwdCfg {
  static constexpr int BM = 128, BN = 128;
  // Q stays until dK of its block, one block longer than S needs it: two stages at least.  dO is released by dV,
  // before dP of the next block needs the next one, so one stage does where shared memory is short.
  static constexpr int QS = (D == 64) ? 3 : 2;
  static constexpr int DS = (D == 64) ? 3 : 1;
  static constexpr bool DQ_ALIAS = (D == 128);          // dQ takes the dP columns
  static constexpr int ATOMS = D / 64;
  static constexpr int ATOM_BYTES = 128 * 128;
  static constexpr int TILE_BYTES = ATOMS * ATOM_BYTES;
  static constexpr int OFF_K = 0;
  static constexpr int OFF_V = OFF_K + TILE_BYTES;
  static constexpr int OFF_Q = OFF_V + TILE_BYTES;              // [QS]
  static constexpr int OFF_DO = OFF_Q + QS * TILE_BYTES;        // [DS]
  static constexpr int OFF_DS = OFF_DO + DS * TILE_BYTES;
  static constexpr int STG_BYTES = 32 * 32 * 4;                 // one 32 x 32 chunk of dQ; two per drain warp
  static constexpr int OFF_STG = OFF_DS + 2 * ATOM_BYTES;
  static constexpr int OFF_ST = OFF_STG + 8 * STG_BYTES;        // [QS] row statistics of a query block
  static constexpr int OFF_BAR = OFF_ST + QS * 1024;
  static constexpr int SMEM = OFF_BAR + 256;
  static constexpr int NBAR = 1 + 2 * QS + 2 * DS + 6;
  static constexpr int NTHREADS = 512;
  // Registers per thread: loads and MMAs / math / drain, which holds a whole row of dQ so that its columns are free at once.
  // (Spills by -Xptxas -v: 24 bytes stored and 160 loaded per thread at d = 64, 76 and 100 at d = 128.)
  static constexpr int REGS_ISSUE = 96, REGS_MATH = (D == 64) ? 160 : 128, REGS_DRAIN = (D == 64) ? 96 : 160;
  static_assert(REGS_ISSUE + 2 * REGS_MATH + REGS_DRAIN <= 4 * 128, "a CTA has 512 x 128 registers");
  // TMEM columns
  static constexpr int COL_S = 0, COL_DP = 128, COL_DV = 256, COL_DK = 256 + D;
  static constexpr int COL_DQ = DQ_ALIAS ? COL_DP : 384;
};
static_assert(BwdCfg<128>::SMEM <= 232448, "shared memory of a CTA");

// First 128-query block that sees key block `nblk`, and the parts that its loop is cut into.
__host__ __device__ __forceinline__ int bwd_first_block(int causal, int nblk, int off) {
  const int first_row = nblk * 128 - off;
  return causal && first_row > 0 ? first_row / 128 : 0;
}
__host__ __device__ __forceinline__ int bwd_parts(int mb_first, int n_mblocks, int rep, int chunk) {
  const int its = (n_mblocks > mb_first ? n_mblocks - mb_first : 0) * rep;
  return its ? (its + chunk - 1) / chunk : 1;      // (one without work where no query sees the block)
}
constexpr int MAX_CUT_BLOCKS = 1024;      // key blocks of a launch in parts

// fp32 accumulator layout: dQ tile (b, h, block of 128 rows), or dK / dV tile of a part -> 4 row quads -> D / 4 pieces of 4 columns -> 32 rows: the 16-byte stores of a
// drain warp (a row per lane) are contiguous, and so are the 16-byte loads of a warp here.  A thread converts 32 columns of a row of dQ, or adds the parts of COLS
// columns of dK or dV (0: the launch was not in parts), 64 / COLS of them loaded at a time.  With few tiles their parts are one chain of loads, shorter the more are in
// flight; with many, the wider pieces of rows count (COLS 8 / 16, backward, graph, us: 1 x 128, 16 / 1 heads, d 64 12.0 / 13.2, 1290 x 130, 16 / 2, d 64 20.9 / 22.7; 4
// x 500, 16 / 4, d 64 28.3 / 26.4, 1 x 8192, 8 / 2, d 128 373 / 367).
template <int D, int COLS>
__global__ void fa_dq_convert_kernel(const FaBwdParams p) {
  grid_go();
  grid_wait();
  const long long threads = (long long)gridDim.x * blockDim.x;
  long long start = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if constexpr (COLS > 0) {
    const int lane = threadIdx.x & 31;
    constexpr int G = D / COLS, U = 64 / COLS, V = COLS / 4;      // U * V 16-byte loads in flight
    const int off = p.Sk - p.Sq, n_mblocks = (p.Sq + 127) / 128, n_nblk = (p.Sk + 127) / 128, rep = p.hq / p.hkv, pairs = p.hkv * p.B;
    __shared__ int s_first[MAX_CUT_BLOCKS + 1];                // parts ahead of a key block's
    if (threadIdx.x < 32) {
      int run = 0;
      for (int k0 = 0; k0 <= n_nblk; k0 += 32) {
        const int k = k0 + lane, own = k < n_nblk ? bwd_parts(bwd_first_block(p.causal, k, off), n_mblocks, rep, p.chunk) : 0;
        int upto = own;                                        // inclusive sum over the lanes
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int v = __shfl_up_sync(0xffffffffu, upto, o);
          if (lane >= o) upto += v;
        }
        if (k <= n_nblk) s_first[k] = run + upto - own;
        run += __shfl_sync(0xffffffffu, upto, 31);
      }
    }
    __syncthreads();
    const int pieces = 2 * pairs * n_nblk * 4 * G;             // (bwd_chunk() cuts launches of few key blocks)
    for (; start < 32LL * pieces; start += threads) {          // (dK or dV, key block, pair, quad, COLS columns)
      const int w = (int)(start >> 5), g = w % G, quad = (w / G) & 3, tile = w / (4 * G);
      const int pair = tile % pairs, block = (tile / pairs) % n_nblk, dv = tile / pairs / n_nblk;
      const int row = block * 128 + quad * 32 + lane;
      if (row >= p.Sk) continue;
      // (CTA part * pairs + pair has left its tile at that index; a block that no query sees has one part, which leaves nothing)
      const int first = s_first[block], end = n_mblocks > bwd_first_block(p.causal, block, off) ? s_first[block + 1] : first;
      const float4* from = reinterpret_cast<const float4*>(dv ? p.dv_acc : p.dk_acc) + (quad * (D / 4) + V * g) * 32 + lane;
      float f[COLS];
#pragma unroll
      for (int i = 0; i < COLS; i++) f[i] = 0.f;
      for (int part = first; part < end; part += U) {
        float4 x[U][V];
#pragma unroll
        for (int u = 0; u < U; u++) {
          const float4* tile_at = from + ((long long)(part + u) * pairs + pair) * (32 * D);
#pragma unroll
          for (int k = 0; k < V; k++)
            if (part + u < end) x[u][k] = tile_at[k * 32];
        }
#pragma unroll
        for (int u = 0; u < U; u++)
          if (part + u < end) {
#pragma unroll
            for (int k = 0; k < V; k++) { f[4 * k] += x[u][k].x; f[4 * k + 1] += x[u][k].y; f[4 * k + 2] += x[u][k].z; f[4 * k + 3] += x[u][k].w; }
          }
      }
      bf16* o = (dv ? p.dv : p.dk) + ((long long)(pair / p.hkv) * p.Sk + row) * (dv ? p.dv_ts : p.dk_ts) + (pair % p.hkv) * D + g * COLS;
#pragma unroll
      for (int k = 0; k < COLS / 8; k++) *reinterpret_cast<uint4*>(o + k * 8) = pack8(f + k * 8);
    }
    start -= 32LL * pieces;                                    // dQ's pieces come next
  }
  constexpr int CPR = D / 32;                                  // 32-column chunks per row
  const int n_mblocks = (p.Sq + 127) / 128;
  const long long total = (long long)p.B * p.hq * n_mblocks * 128 * CPR;
  for (long long idx = start; idx < total; idx += threads) {
    const int lane = (int)(idx & 31);
    const long long w = idx >> 5;                              // (tile, quad, chunk): the accumulator's order
    const int chunk = (int)(w % CPR), quad = (int)((w / CPR) & 3);
    const long long tile = w / (CPR * 4);
    const int mblock = (int)(tile % n_mblocks);
    const long long bh = tile / n_mblocks;
    const int row = mblock * 128 + quad * 32 + lane;
    if (row >= p.Sq) continue;
    const int h = (int)(bh % p.hq);
    const long long b = bh / p.hq;
    const float4* at = reinterpret_cast<const float4*>(p.dq_acc) + (w * 8) * 32 + lane;
    float f[32];
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const float4 v = at[k * 32];
      f[4 * k] = v.x; f[4 * k + 1] = v.y; f[4 * k + 2] = v.z; f[4 * k + 3] = v.w;
    }
    bf16* o = p.dq + (b * p.Sq + row) * p.dq_ts + (long long)h * D + chunk * 32;
#pragma unroll
    for (int k = 0; k < 4; k++) *reinterpret_cast<uint4*>(o + k * 8) = pack8(f + k * 8);
  }
}

// Row statistics, one 1 KB record per (b, h, 128-query block): 128 x -lse * log2(e), then 128 x -scale * sum_d o * do.  Rows
// past Sq get (-inf, 0), which makes their P and dS zero.  Also clears dQ's accumulator.  D/8 threads per (token, head).
template <int D>
__global__ void fa_bwd_prep_kernel(const FaBwdParams p) {
  grid_go();
  grid_wait();
  constexpr int TPR = D / 8;                                   // threads per row: 8 or 16
  const int n_mblocks = (p.Sq + 127) / 128, Sp = n_mblocks * 128;
  const long long total = (long long)p.B * Sp * p.hq;
  const int rpb = blockDim.x / TPR;                            // rows per block and iteration
  const int sub = threadIdx.x % TPR;
  // every thread of the block runs the same number of iterations, so the shuffles see whole warps
  for (long long base = (long long)blockIdx.x * rpb; base < total; base += (long long)gridDim.x * rpb) {
    const long long idx = base + threadIdx.x / TPR;
    const bool live = idx < total;
    float s = 0.f;
    int h = 0, b = 0, i = 0;
    if (live) {
      h = (int)(idx % p.hq);
      const long long bi = idx / p.hq;
      b = (int)(bi / Sp);
      i = (int)(bi % Sp);
      if (!p.alone) {
        float4* z = reinterpret_cast<float4*>(p.dq_acc + (idx * TPR + sub) * 8);
        z[0] = make_float4(0.f, 0.f, 0.f, 0.f);
        z[1] = make_float4(0.f, 0.f, 0.f, 0.f);
      }
      if (i < p.Sq) {
        const long long row = (long long)b * p.Sq + i;
        float a[8], e[8];
        unpack8(*reinterpret_cast<const uint4*>(p.o + row * p.o_ts + (long long)h * D + sub * 8), a);
        unpack8(*reinterpret_cast<const uint4*>(p.dout + row * p.do_ts + (long long)h * D + sub * 8), e);
#pragma unroll
        for (int k = 0; k < 8; k++) s += a[k] * e[k];
      }
    }
#pragma unroll
    for (int o = TPR / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);   // whole warps stay converged
    if (live && sub == 0) {
      float* rec = p.stats + (((long long)b * p.hq + h) * n_mblocks + (i >> 7)) * 256 + (i & 127);
      rec[0] = i < p.Sq ? -p.lse[((long long)b * p.hq + h) * p.Sq + i] * 1.4426950408889634f : -INFINITY;
      rec[128] = -s * p.scale;
    }
  }
}

// What a CTA leaves: WHOLE dK and dV of a key block, and its share of dQ, added to the fp32 sums; PARTS (with chunk) that, and its share of dK and dV; ALONE
// all three.
enum : int { WHOLE, PARTS_OF, ALONE };
template <int D, int FORM>
__global__ void __launch_bounds__(512, 1)
fa_bwd_tc_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk,
                 const __grid_constant__ CUtensorMap tv, const __grid_constant__ CUtensorMap tdo, const __grid_constant__ CUtensorMap tdo_end, const __grid_constant__ CUtensorMap tdk,
                 const __grid_constant__ CUtensorMap tdv, const FaBwdParams p) {
  using C = BwdCfg<D>;
  constexpr bool PARTS = FORM == PARTS_OF;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::OFF_BAR);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + C::NBAR);
  int* s_abort = reinterpret_cast<int*>(tmem_slot + 1);     // {abort, extra wait in ms}: see bw::mbar_wait

  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;   // (uniform over the warp)
  const uint32_t sbase = smem_u32(smem);
  if (sbase & 1023u) {                                       // the swizzled tiles need it; nothing has been started yet
    if (threadIdx.x == 0) atomicExch(&g_fab_status[0], 4u);
    return;
  }
  const uint32_t bar0 = smem_u32(bars);
  const uint32_t kv_full = bar0;
  auto q_full = [&](int s) { return bar0 + 8u * (1 + s); };
  auto q_empty = [&](int s) { return bar0 + 8u * (1 + C::QS + s); };
  auto do_full = [&](int s) { return bar0 + 8u * (1 + 2 * C::QS + s); };
  auto do_empty = [&](int s) { return bar0 + 8u * (1 + 2 * C::QS + C::DS + s); };
  const uint32_t bar1 = bar0 + 8u * (1 + 2 * C::QS + 2 * C::DS);
  const uint32_t s_full = bar1, dp_full = bar1 + 8, p_full = bar1 + 16, ds_full = bar1 + 24, dq_full = bar1 + 32, dq_free = bar1 + 40;

  // 1-D grid.  Under a causal mask the first key block is seen by every query and the last by one block,
  // so the CTAs of early key blocks of all (batch, kv head) pairs of a group come first (longest first: with
  // one pair after the other, the last pair's longest CTA started when the chip was almost done).  In parts: those of the first key block of all
  // pairs, then the next.
  const int n_nblk = (p.Sk + C::BN - 1) / C::BN;
  int nblk, pair, it_first = 0;
  if constexpr (PARTS) {
    const int pairs = p.hkv * p.B;
    pair = (int)blockIdx.x % pairs;
    int part = (int)blockIdx.x / pairs;
    for (nblk = 0; nblk + 1 < n_nblk; nblk++) {
      const int parts = bwd_parts(bwd_first_block(p.causal, nblk, p.Sk - p.Sq), (p.Sq + C::BM - 1) / C::BM, p.hq / p.hkv, p.chunk);
      if (part < parts) break;
      part -= parts;
    }
    it_first = part * p.chunk;
  } else {
    const int grp = (int)blockIdx.x / (n_nblk * BWD_GROUP);
    const int in_grp = (int)blockIdx.x - grp * n_nblk * BWD_GROUP;
    const int gsize = min(BWD_GROUP, p.hkv * p.B - grp * BWD_GROUP);
    nblk = in_grp / gsize;
    pair = grp * BWD_GROUP + in_grp % gsize;
  }
  const int hk = pair % p.hkv, b = pair / p.hkv;
  const int n0 = nblk * C::BN;
  const int off = p.Sk - p.Sq;
  const int rep = p.hq / p.hkv;
  const int n_mblocks = (p.Sq + C::BM - 1) / C::BM;
  int mb_first = 0;
  if (p.causal) {
    const int first_row = n0 - off;
    mb_first = first_row > 0 ? first_row / C::BM : 0;
  }
  const int per_head = n_mblocks > mb_first ? n_mblocks - mb_first : 0;
  // query blocks of every head of the group, head by head; a part takes `chunk` of them
  const int total_it = PARTS ? min(p.chunk, per_head * rep - it_first) : per_head * rep;
  const int h_first = hk * rep + (PARTS && per_head ? it_first / per_head : 0), mb_start = mb_first + (PARTS && per_head ? it_first % per_head : 0);

  if (threadIdx.x == 0) {
    s_abort[0] = 0;
    s_abort[1] = 0;
    mbar_init(kv_full, 1);
    for (int s = 0; s < C::QS; s++) { mbar_init(q_full(s), 1); mbar_init(q_empty(s), 1); }
    for (int s = 0; s < C::DS; s++) { mbar_init(do_full(s), 1); mbar_init(do_empty(s), 1); }
    mbar_init(s_full, 1);
    mbar_init(dp_full, 1);
    mbar_init(p_full, 8);
    mbar_init(ds_full, 8);
    mbar_init(dq_full, 1);
    mbar_init(dq_free, 4);
    mbar_init_fence();
    prefetch_tmap(&tq); prefetch_tmap(&tk); prefetch_tmap(&tv); prefetch_tmap(&tdo); prefetch_tmap(&tdk); prefetch_tmap(&tdv);
  }
  if (warp == 1) tmem_alloc(smem_u32(tmem_slot), 512);
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  volatile int* abort_flag = s_abort;
  grid_wait();

  if (warp < 4) reg_dec<C::REGS_ISSUE>();
  if (warp == 0) {
    // ------------------------------- TMA producer -------------------------------
    if (total_it > 0 && elect_one()) {
      mbar_expect_tx(kv_full, 2 * C::TILE_BYTES);
#pragma unroll
      for (int a = 0; a < C::ATOMS; a++) {
        tma_load_3d(sbase + C::OFF_K + a * C::ATOM_BYTES, &tk, hk * D + a * 64, n0, b, kv_full);
        tma_load_3d(sbase + C::OFF_V + a * C::ATOM_BYTES, &tv, hk * D + a * 64, n0, b, kv_full);
      }
      bool ok = true;
      const int ragged = p.Sq % C::BM ? n_mblocks - 1 : -1;
      int h = h_first, mb = mb_start, st = 0, dst = 0;
      uint32_t ph = 1u, dph = 1u;
      for (int it = 0; it < total_it; it++) {
        if (!mbar_wait(q_empty(st), ph, abort_flag)) { ok = false; break; }
        mbar_expect_tx(q_full(st), C::TILE_BYTES + 1024);
#pragma unroll
        for (int a = 0; a < C::ATOMS; a++)
          tma_load_3d(sbase + C::OFF_Q + st * C::TILE_BYTES + a * C::ATOM_BYTES, &tq, h * D + a * 64, mb * C::BM, b, q_full(st));
        bulk_load(sbase + C::OFF_ST + st * 1024, p.stats + (((long long)b * p.hq + h) * n_mblocks + mb) * 256, 1024, q_full(st));
        if (!mbar_wait(do_empty(dst), dph, abort_flag)) { ok = false; break; }
        mbar_expect_tx(do_full(dst), C::TILE_BYTES);
#pragma unroll
        for (int a = 0; a < C::ATOMS; a++)
          if (mb == ragged) tma_load_3d(sbase + C::OFF_DO + dst * C::TILE_BYTES + a * C::ATOM_BYTES, &tdo_end, h * D + a * 64, mb * C::BM, b, do_full(dst));
          else tma_load_2d(sbase + C::OFF_DO + dst * C::TILE_BYTES + a * C::ATOM_BYTES, &tdo, h * D + a * 64, b * p.Sq + mb * C::BM, do_full(dst));
        if (++mb == n_mblocks) { mb = mb_first; h++; }
        if (++st == C::QS) { st = 0; ph ^= 1u; }
        if (++dst == C::DS) { dst = 0; dph ^= 1u; }
      }
      if (!ok) atomicExch(&g_fab_status[0], 1u);
    }
  } else if (warp == 1) {
    // ------------------------------- MMA issuer -------------------------------
    if (total_it > 0 && elect_one()) {
      const uint32_t idesc_s = make_idesc(128, 128, 0, 0);     // S^T, dP^T: K-major A and B
      const uint32_t idesc_kv = make_idesc(128, D, 0, 1);      // dV, dK: A in TMEM, MN-major B
      const uint32_t idesc_dq = make_idesc(128, D, 1, 1);      // dQ: MN-major A and B
      // descriptor bases; a stage / k-step only changes the 16-byte-granular start address
      const uint64_t kK = make_desc(sbase + C::OFF_K, 16, 1024), kV = make_desc(sbase + C::OFF_V, 16, 1024);
      const uint64_t kQ = make_desc(sbase + C::OFF_Q, 16, 1024), kDO = make_desc(sbase + C::OFF_DO, 16, 1024);
      const uint64_t mK = make_desc(sbase + C::OFF_K, C::ATOM_BYTES, 1024), mDS = make_desc(sbase + C::OFF_DS, C::ATOM_BYTES, 1024);
      const uint64_t mQ = make_desc(sbase + C::OFF_Q, C::ATOM_BYTES, 1024), mDO = make_desc(sbase + C::OFF_DO, C::ATOM_BYTES, 1024);
      auto scores = [&](int col, uint64_t a, uint64_t bq) {      // [128 keys x 128 queries] over d
#pragma unroll
        for (int s = 0; s < D / 16; s++) {
          const uint64_t o = (uint64_t)(((s >> 2) * C::ATOM_BYTES + (s & 3) * 32) >> 4);
          umma_bf16(tmem_base + col, a + o, bq + o, idesc_s, s ? 1u : 0u);
        }
      };
      // A (P^T or dS^T): 16 queries of a warpgroup's 64 are 8 columns; the second warpgroup's start 64 columns on
      auto grad_kv = [&](int col, int acol, uint64_t bop, uint32_t acc) {
#pragma unroll
        for (int s = 0; s < C::BM / 16; s++)
          umma_bf16_ta(tmem_base + col, tmem_base + acol + (s >> 2) * 64 + (s & 3) * 8, bop + (uint64_t)(s * 128), idesc_kv,
                       s ? 1u : acc);
      };
      // What a step waits for is waited for ahead of the wait that is the last to come: a wait takes some 100 cycles even where
      // there is nothing to wait for.
      auto issue_s = [&](uint64_t so) {                          // (Q is there)
        scores(C::COL_S, kK, kQ + so);
        umma_commit(s_full);
      };
      auto issue_dp = [&](uint64_t so) {                         // (dO is there, dQ has left the columns)
        scores(C::COL_DP, kV, kDO + so);
        umma_commit(dp_full);
      };
      bool ok = mbar_wait(kv_full, 0, abort_flag) && mbar_wait(q_full(0), 0, abort_flag);
      if (ok) { fence_after(); issue_s(0); ok = mbar_wait(do_full(0), 0, abort_flag); }
      if (ok) { fence_after(); issue_dp(0); }
      int st = 0, dst = 0;
      uint32_t ph = 0, dph = 0;
      for (int it = 0; it < total_it && ok; it++) {
        const bool more = it + 1 < total_it;
        const int sn = st + 1 == C::QS ? 0 : st + 1, dn = dst + 1 == C::DS ? 0 : dst + 1;       // stages of the next block
        const uint32_t phn = sn ? ph : ph ^ 1u, dphn = dn ? dph : dph ^ 1u;
        if (more && !(ok = mbar_wait(q_full(sn), phn, abort_flag))) break;
        if (!(ok = mbar_wait(p_full, (uint32_t)it & 1u, abort_flag))) break;
        fence_after();
        grad_kv(C::COL_DV, C::COL_S, mDO + (uint64_t)((dst * C::TILE_BYTES) >> 4), it ? 1u : 0u);       // dV += P^T dO
        umma_commit(do_empty(dst));
        if (more) issue_s((uint64_t)((sn * C::TILE_BYTES) >> 4));        // P^T has been read: S^T of the next block
        if (!C::DQ_ALIAS && more && !(ok = mbar_wait(do_full(dn), dphn, abort_flag))) break;
        if (!C::DQ_ALIAS && it > 0 && !(ok = mbar_wait(dq_free, (uint32_t)(it - 1) & 1u, abort_flag))) break;
        if (!(ok = mbar_wait(ds_full, (uint32_t)it & 1u, abort_flag))) break;
        fence_after();
        grad_kv(C::COL_DK, C::COL_DP, mQ + (uint64_t)((st * C::TILE_BYTES) >> 4), it ? 1u : 0u);        // dK += dS^T Q
        umma_commit(q_empty(st));
        if (!C::DQ_ALIAS && more) issue_dp((uint64_t)((dn * C::TILE_BYTES) >> 4));
#pragma unroll
        for (int s = 0; s < C::BN / 16; s++)                             // dQ = dS K
          umma_bf16(tmem_base + C::COL_DQ, mDS + (uint64_t)(s * 128), mK + (uint64_t)(s * 128), idesc_dq, s ? 1u : 0u);
        umma_commit(dq_full);
        if (C::DQ_ALIAS && more) {
          if (!(ok = mbar_wait(do_full(dn), dphn, abort_flag))) break;
          if (!(ok = mbar_wait(dq_free, (uint32_t)it & 1u, abort_flag))) break;
          fence_after();
          issue_dp((uint64_t)((dn * C::TILE_BYTES) >> 4));
        }
        st = sn; ph = phn;
        dst = dn; dph = dphn;
      }
      if (!ok) atomicExch(&g_fab_status[0], 2u);
    }
  } else if (warp >= 12) {
    if constexpr (C::REGS_DRAIN > 128) reg_inc<C::REGS_DRAIN>(); else reg_dec<C::REGS_DRAIN>();
    // ------------------------------- dQ drain -------------------------------
    const int quad = warp & 3;
    const uint32_t tdq = tmem_base + ((uint32_t)(quad * 32) << 16) + C::COL_DQ;
    uint8_t* stg = smem + C::OFF_STG + quad * 2 * C::STG_BYTES;
    [[maybe_unused]] float* tile = p.dq_acc + (((long long)b * p.hq + h_first) * n_mblocks + mb_start) * (128 * D) + quad * (32 * D);
    bool ok = true;
    int mb = mb_start;
    for (int it = 0; it < total_it; it++) {
      if (!mbar_wait(dq_full, (uint32_t)it & 1u, abort_flag)) { ok = false; break; }
      fence_after();
      uint32_t r[D];
#pragma unroll
      for (int c = 0; c < D / 32; c++) tmem_ld32(tdq + c * 32, r + c * 32);
      tmem_ld_wait();
      fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(dq_free);
      if constexpr (FORM == ALONE) {
        // the query block's dQ is complete: a row per lane
        const int row = mb * C::BM + quad * 32 + lane;
        if (row < p.Sq) {
          bf16* o = p.dq + ((long long)b * p.Sq + row) * p.dq_ts + (long long)(h_first + it / n_mblocks) * D;
#pragma unroll
          for (int k = 0; k < D / 8; k++) *reinterpret_cast<uint4*>(o + k * 8) = pack8(reinterpret_cast<const float*>(r) + k * 8);
        }
        if (++mb == n_mblocks) mb = 0;
      } else {
#pragma unroll
        for (int c = 0; c < D / 32; c++) {
          uint8_t* sp = stg + (c & 1) * C::STG_BYTES;
          if (lane == 0) bulk_wait_read_but<1>();      // this half of the staging has been read
          __syncwarp();
#pragma unroll
          for (int k = 0; k < 8; k++)
            *reinterpret_cast<uint4*>(sp + k * 512 + lane * 16) =
                make_uint4(r[c * 32 + k * 4], r[c * 32 + k * 4 + 1], r[c * 32 + k * 4 + 2], r[c * 32 + k * 4 + 3]);
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            bulk_reduce_add_f32(tile + c * 1024, smem_u32(sp), C::STG_BYTES);
            bulk_commit();
          }
        }
        tile += 128 * D;
        if (++mb == n_mblocks) { mb = mb_first; tile += (long long)mb_first * (128 * D); }
      }
    }
    if (lane == 0) bulk_wait_read_but<0>();
    if (!ok && lane == 0) atomicExch(&g_fab_status[0], 5u);
  } else if (warp >= 4) {
    reg_inc<C::REGS_MATH>();
    // ------------------------------- math warps -------------------------------
    const int quad = warp & 3;
    const int wg = (warp - 4) >> 2;                 // which 64 of the 128 query columns
    const int rit = quad * 32 + lane;               // key row inside the block
    const int key = n0 + rit;
    const uint32_t lane_addr = tmem_base + ((uint32_t)(quad * 32) << 16);
    const uint32_t ts = lane_addr + C::COL_S + wg * 64, tdp = lane_addr + C::COL_DP + wg * 64;
    const f32x2 sl2 = pack2(p.scale * 1.4426950408889634f, p.scale * 1.4426950408889634f);
    const f32x2 sc = pack2(p.scale, p.scale);
    uint8_t* sds = smem + C::OFF_DS + wg * C::ATOM_BYTES;
    bool ok = true;
    int mb = mb_start, qs = 0;
    uint32_t qph = 0;
    for (int it = 0; it < total_it; it++) {
      const int m0 = mb * C::BM;
      const float4* st = reinterpret_cast<const float4*>(smem + C::OFF_ST + qs * 1024) + wg * 16;
      if (!mbar_wait(q_full(qs), qph, abort_flag) ||        // the statistics
          !mbar_wait(s_full, (uint32_t)it & 1u, abort_flag)) { ok = false; break; }
      fence_after();
      float pf[64];
      {
        uint32_t sr[64];
        tmem_ld32(ts, sr);
        tmem_ld32(ts + 32, sr + 32);
        tmem_ld_wait();
        // P^T of this key and 64 queries; the key is seen by queries lo and later of this block
        const bool need_mask = (n0 + C::BN > p.Sk) || (p.causal && m0 + off < n0 + quad * 32 + 31);
        const int lo = (key >= p.Sk ? 1 << 20 : (p.causal ? key - off - m0 : 0)) - wg * 64;
#pragma unroll
        for (int c = 0; c < 16; c++) {
          const float4 nl = st[c];
          float x[4];
          unpack2(fma2(pack2(__uint_as_float(sr[c * 4]), __uint_as_float(sr[c * 4 + 1])), sl2, pack2(nl.x, nl.y)), x[0], x[1]);
          unpack2(fma2(pack2(__uint_as_float(sr[c * 4 + 2]), __uint_as_float(sr[c * 4 + 3])), sl2, pack2(nl.z, nl.w)), x[2], x[3]);
#pragma unroll
          for (int k = 0; k < 4; k++) pf[c * 4 + k] = exp2f(x[k]);
        }
        if (need_mask) {
#pragma unroll
          for (int i = 0; i < 64; i++)
            if (i < lo) pf[i] = 0.f;
        }
      }
      {
        uint32_t pp[32];
#pragma unroll
        for (int i = 0; i < 32; i++) {
          bf162 pb = __floats2bfloat162_rn(pf[2 * i], pf[2 * i + 1]);
          pp[i] = *reinterpret_cast<uint32_t*>(&pb);
        }
        tmem_st32(ts, pp);
        tmem_st_wait();
      }
      fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full);
      if (!mbar_wait(dp_full, (uint32_t)it & 1u, abort_flag)) { ok = false; break; }
      fence_after();
      uint32_t dd[32];
#pragma unroll
      for (int half = 0; half < 2; half++) {
        uint32_t dr[32];
        tmem_ld32(tdp + half * 32, dr);
        tmem_ld_wait();
#pragma unroll
        for (int c = 0; c < 8; c++) {
          const float4 nd = st[32 + half * 8 + c];
          const int i = half * 32 + c * 4;
          const f32x2 d01 = mul2(pack2(pf[i], pf[i + 1]),
                                 fma2(pack2(__uint_as_float(dr[c * 4]), __uint_as_float(dr[c * 4 + 1])), sc, pack2(nd.x, nd.y)));
          const f32x2 d23 = mul2(pack2(pf[i + 2], pf[i + 3]),
                                 fma2(pack2(__uint_as_float(dr[c * 4 + 2]), __uint_as_float(dr[c * 4 + 3])), sc, pack2(nd.z, nd.w)));
          float d[4];
          unpack2(d01, d[0], d[1]);
          unpack2(d23, d[2], d[3]);
          bf162 a = __floats2bfloat162_rn(d[0], d[1]), e = __floats2bfloat162_rn(d[2], d[3]);
          dd[i >> 1] = *reinterpret_cast<uint32_t*>(&a);
          dd[(i >> 1) + 1] = *reinterpret_cast<uint32_t*>(&e);
        }
      }
      tmem_st32(tdp, dd);
      // the shared copy may be rewritten once dQ of the previous block has read it
      if (it > 0 && !mbar_wait(dq_full, (uint32_t)(it - 1) & 1u, abort_flag)) { ok = false; break; }
#pragma unroll
      for (int c = 0; c < 8; c++)
        *reinterpret_cast<uint4*>(sds + sw128_off(rit, c)) = make_uint4(dd[c * 4], dd[c * 4 + 1], dd[c * 4 + 2], dd[c * 4 + 3]);
      tmem_st_wait();
      fence_before();
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(ds_full);
      if (++mb == n_mblocks) mb = mb_first;
      if (++qs == C::QS) { qs = 0; qph ^= 1u; }
    }
    // dQ of the last block is the last MMA: everything has finished
    if (ok && total_it > 0) ok = mbar_wait(dq_full, (uint32_t)(total_it - 1) & 1u, abort_flag);
    if (PARTS && ok && total_it > 0) {
      // to this CTA's place, 32 columns at a time
      fence_after();
      float* sum = (wg ? p.dk_acc : p.dv_acc) + (long long)blockIdx.x * (128 * D) + quad * (32 * D);
      uint8_t* out = smem + (wg ? C::OFF_V : C::OFF_K) + quad * C::STG_BYTES;
#pragma unroll 1
      for (int c = 0; c < D / 32; c++) {
        uint32_t r[32];
        tmem_ld32(lane_addr + (wg ? C::COL_DK : C::COL_DV) + c * 32, r);
        tmem_ld_wait();
        if (lane == 0) bulk_wait_read_but<0>();
        __syncwarp();
#pragma unroll
        for (int k = 0; k < 8; k++)
          *reinterpret_cast<uint4*>(out + k * 512 + lane * 16) = make_uint4(r[k * 4], r[k * 4 + 1], r[k * 4 + 2], r[k * 4 + 3]);
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          bulk_store(sum + c * 1024, smem_u32(out), C::STG_BYTES);
          bulk_commit();
        }
      }
      if (lane == 0) bulk_wait_read_but<0>();        // nothing reads shared memory after the CTA's end
    } else if (!PARTS && ok && total_it > 0) {
      // through shared memory (K's tile for dV, V's for dK: nothing reads them any more), 64 columns of 32 keys at a time
      fence_after();
#pragma unroll 1
      for (int a = 0; a < C::ATOMS; a++) {
        uint8_t* out = smem + (wg ? C::OFF_V : C::OFF_K) + a * C::ATOM_BYTES + quad * 4096;
        uint32_t r[64];
        tmem_ld32(lane_addr + (wg ? C::COL_DK : C::COL_DV) + a * 64, r);
        tmem_ld32(lane_addr + (wg ? C::COL_DK : C::COL_DV) + a * 64 + 32, r + 32);
        tmem_ld_wait();
#pragma unroll
        for (int g = 0; g < 8; g++) {
          float f[8];
#pragma unroll
          for (int i = 0; i < 8; i++) f[i] = __uint_as_float(r[g * 8 + i]);
          *reinterpret_cast<uint4*>(out + sw128_off(lane, g)) = pack8(f);
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0 && n0 + quad * 32 < p.Sk) {
          tma_store_3d(wg ? &tdk : &tdv, smem_u32(out), hk * D + a * 64, n0 + quad * 32, b);
          bulk_commit();
        }
      }
      if (lane == 0) bulk_wait_read_but<0>();        // nothing reads shared memory after the CTA's end
    } else if (!PARTS && total_it == 0 && key < p.Sk) {
      // no query sees these keys: their gradients are zero
      bf16* orow = wg ? p.dk + ((long long)b * p.Sk + key) * p.dk_ts + (long long)hk * D
                      : p.dv + ((long long)b * p.Sk + key) * p.dv_ts + (long long)hk * D;
      for (int c = 0; c < D / 8; c++) *reinterpret_cast<uint4*>(orow + c * 8) = make_uint4(0, 0, 0, 0);
    }
    if (!ok && lane == 0) atomicExch(&g_fab_status[0], 3u);
  }

  fence_before();
  __syncthreads();
  if (warp == 1) {
    fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// CTAs of a launch in parts of `chunk` query blocks.
long long bwd_ctas(int B, int Sq, int Sk, int hq, int hkv, int causal, int chunk) {
  const int n_mblocks = (Sq + 127) / 128, rep = hq / hkv;
  long long n = 0;
  for (int k = 0; k < (Sk + 127) / 128; k++) n += bwd_parts(bwd_first_block(causal, k, Sk - Sq), n_mblocks, rep, chunk);
  return n * hkv * B;
}
// Query blocks of a part, or 0 where a CTA per key block is modelled to be as good.  In query blocks: a CTA's fixed part is some 6, leaving
// dK / dV in fp32 instead of writing them 3 and their conversion 2 more.  Whole / parts, us, all kernels, causal: B2 S2000 16q/2kv d64 258 / 92, B1 S2000
// 16q/4kv d64 116 / 51 and d128 159 / 71, B1 S8192 8q/2kv d128 561 / 365 and 2q/2kv 147 / 116, B4 S500 16q/4kv d64 40 / 28, B1 S300 8q/2kv d64 30 / 14; left
// whole B8 S2048 32q/4kv d64, B1 S8192 32q/8kv d128, B3 S1531 32q/8kv d128, B2 S1728 4q/4kv d64.
// (Measured with parts that added to one sum as they came.  Places of their own, whose order is fixed, against that, backward as graphs: B2 S2000 16q/2kv d64 81.0 / 82.4,
// B1 S2000 16q/4kv d128 66.2 / 69.2, B1 S8192 8q/2kv d128 360 / 367 and 2q/2kv 114 / 120, B4 S500 16q/4kv d64 25.4 / 26.4, B1 S300 8q/2kv d64 11.9 / 12.0.)
int bwd_chunk(int B, int Sq, int Sk, int hq, int hkv, int causal, int sms) {
  const int n_mblocks = (Sq + 127) / 128, n_nblk = (Sk + 127) / 128, rep = hq / hkv, pairs = hkv * B;
  if ((long long)n_nblk * pairs > 4LL * sms || n_nblk > MAX_CUT_BLOCKS) return 0;      // (several CTAs per SM, longest first)
  long long total = 0, longest = 0;
  for (int k = 0; k < n_nblk; k++) {
    const long long its = (long long)std::max(0, n_mblocks - bwd_first_block(causal, k, Sk - Sq)) * rep;
    total += (its + 6) * pairs;
    longest = std::max(longest, its + 6);
  }
  const double whole = std::max((double)longest, 1.1 * (double)total / sms);
  int best = 0;
  double best_time = 0.9 * whole;
  for (int waves = 1; waves <= 2; waves++) {
    // the smallest parts that make no more CTAs than that many per SM
    int lo = 1, hi = n_mblocks * rep;
    while (lo < hi) {
      const int mid = (lo + hi) / 2;
      if (bwd_ctas(B, Sq, Sk, hq, hkv, causal, mid) <= (long long)waves * sms) hi = mid; else lo = mid + 1;
    }
    const double time = waves * (lo + 9.0) + 2.0;
    if (time < best_time && bwd_ctas(B, Sq, Sk, hq, hkv, causal, lo) <= (long long)waves * sms) { best = lo; best_time = time; }
  }
  return best;
}

template <int D>
int launch_fa_bwd(const void* q, const void* k, const void* v, const FaBwdParams& p, long long q_ts, long long k_ts,
                  long long v_ts, cudaStream_t s) {
  using C = BwdCfg<D>;
  CUtensorMap tq, tk, tv, tdo, tdo_end, tdk, tdv;
  int rc;
  // (sequence by sequence: rows past a sequence's last are zeros.  Their P and dS are zero, but zero times what the next sequence holds is not, where
  // that is infinite or NaN.  dO only for blocks that end inside a sequence's tile: a load by the map with a third dimension takes longer, and at d 128 a block
  // waits for dO: 1 x 8192, 32 / 8 heads 1265 us, now 1254.)
  const uint64_t B = p.B, Sq = p.Sq, Sk = p.Sk, brows = p.kv_brows, q_cols = (uint64_t)p.hq * D, kv_cols = (uint64_t)p.hkv * D;
  if ((rc = make_map_bf16_3d(&tq, q, q_cols, Sq, Sq, B, (uint64_t)q_ts, 64, 128))) return rc;
  if ((rc = make_map_bf16_3d(&tk, k, kv_cols, Sk, brows, B, (uint64_t)k_ts, 64, 128))) return rc;
  if ((rc = make_map_bf16_3d(&tv, v, kv_cols, Sk, brows, B, (uint64_t)v_ts, 64, 128))) return rc;
  if ((rc = make_map_bf16(&tdo, p.dout, q_cols, B * Sq, (uint64_t)p.do_ts, 64, 128))) return rc;
  if ((rc = make_map_bf16_3d(&tdo_end, p.dout, q_cols, Sq, Sq, B, (uint64_t)p.do_ts, 64, 128))) return rc;
  if ((rc = make_map_bf16_3d(&tdk, p.dk, kv_cols, Sk, Sk, B, (uint64_t)p.dk_ts, 64, 32))) return rc;
  if ((rc = make_map_bf16_3d(&tdv, p.dv, kv_cols, Sk, Sk, B, (uint64_t)p.dv_ts, 64, 32))) return rc;
  static bool attr = false;
  if (!attr) {
    // the register split must fit in what the launch allocates, or it would wait for registers that nobody gives back
    for (auto fn : {fa_bwd_tc_kernel<D, WHOLE>, fa_bwd_tc_kernel<D, PARTS_OF>, fa_bwd_tc_kernel<D, ALONE>}) {
      cudaFuncAttributes fa;
      if (cudaFuncGetAttributes(&fa, fn) != cudaSuccess || (fa.numRegs + 7) / 8 * 8 != 128) return LB_ERR_LAUNCH;
      cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
    }
    attr = true;
  }
  long long grid = (long long)((p.Sk + 127) / 128) * p.hkv * p.B;
  if (grid > 2147483647LL) return LB_ERR_SHAPE;
  if (p.chunk) grid = bwd_ctas(p.B, p.Sq, p.Sk, p.hq, p.hkv, p.causal, p.chunk);
  const long long rows = (long long)p.B * ((p.Sq + 127) / 128 * 128) * p.hq;
  const long long rows_per_block = 256 / (D / 8), cap = lb_num_sms() * 16;
  const long long pblocks = (rows + rows_per_block - 1) / rows_per_block;
  LB_LAUNCH(fa_bwd_prep_kernel<D>, (int)(pblocks < cap ? pblocks : cap), 256, 0, s, p);
  LB_LAUNCH(p.chunk ? fa_bwd_tc_kernel<D, PARTS_OF> : p.alone ? fa_bwd_tc_kernel<D, ALONE> : fa_bwd_tc_kernel<D, WHOLE>, (unsigned)grid, C::NTHREADS, C::SMEM, s, tq, tk, tv, tdo, tdo_end, tdk, tdv, p);
  if (p.alone) return LB_OK;
  const long long part_rows = p.chunk ? 2LL * p.B * ((p.Sk + 127) / 128 * 128) * p.hkv : 0;
  const int cols = part_rows * (D / 16) < 32 * 4LL * lb_num_sms() ? 8 : 16;      // (16: four warps on an SM have work)
  const long long cblocks = (rows * (D / 32) + part_rows * (D / cols) + 255) / 256;
  LB_LAUNCH(!p.chunk ? fa_dq_convert_kernel<D, 0> : cols == 8 ? fa_dq_convert_kernel<D, 8> : fa_dq_convert_kernel<D, 16>, (int)(cblocks < cap ? cblocks : cap), 256, 0, s, p);
  return LB_OK;
}

}  // namespace

// Copies the status words of the tcgen05 attention backward kernel to host memory and clears them.
extern "C" int lb_flash_bwd_status(void* out) {
  cudaError_t e = cudaMemcpyFromSymbol(out, g_fab_status, sizeof(unsigned int) * 4);
  if (e != cudaSuccess) { g_lb_last_cuda_error = (int)e; return LB_ERR_LAUNCH; }
  unsigned int zeros[4] = {0, 0, 0, 0};
  cudaMemcpyToSymbol(g_fab_status, zeros, sizeof(zeros));
  return LB_OK;
}

// Bytes of the workspace of lb_flash_bwd_tc_ws / lb_flash_bwd_cp_ws: the row statistics (fa_bwd_prep_kernel), then the fp32 dQ
// accumulator (fa_dq_convert_kernel has its layout), both in whole 128-query blocks.  0 for sizes that they do not take.
extern "C" long long lb_flash_bwd_ws_bytes(int B, int Sq, int hq, int d) {
  if (B <= 0 || Sq <= 0 || hq <= 0 || (d != 64 && d != 128)) return 0;
  return (long long)B * hq * ((Sq + 127) / 128) * 128 * (2 + d) * (long long)sizeof(float);
}

// Bytes of one of dk_acc and dv_acc of a launch in parts of `chunk` query blocks, which makes two CTAs per SM at most (39 MB of both, d 128, 148 SMs).
static long long bwd_parts_bytes(int B, int Sq, int Sk, int hq, int hkv, int d, int causal, int chunk) {
  return bwd_ctas(B, Sq, Sk, hq, hkv, causal, chunk) * 128 * d * (long long)sizeof(float);
}

// As above with room for the parts' fp32 dK / dV where the launch is better cut into parts (zero otherwise): what the caller of lb_flash_bwd_tc_ws should bring.
// With lb_flash_bwd_ws_bytes() a CTA takes a whole key block.
extern "C" long long lb_flash_bwd_ws_bytes_kv(int B, int Sq, int Sk, int hq, int hkv, int d, int causal) {
  const long long q = lb_flash_bwd_ws_bytes(B, Sq, hq, d);
  if (!q || Sk <= 0 || hkv <= 0 || hq % hkv) return q;
  const int chunk = bwd_chunk(B, Sq, Sk, hq, hkv, causal, lb_num_sms());
  return chunk ? q + 2 * bwd_parts_bytes(B, Sq, Sk, hq, hkv, d, causal, chunk) : q;
}

// Host only (no CUDA call): query blocks per CTA of the launch for these sizes on `sms` SMs, given that workspace; 0: all of a key block.
extern "C" int lb_flash_bwd_chunk(int B, int Sq, int Sk, int hq, int hkv, int causal, int sms) {
  if (B <= 0 || Sq <= 0 || Sk <= 0 || hq <= 0 || hkv <= 0 || hq % hkv || sms <= 0) return LB_ERR_SHAPE;
  return bwd_chunk(B, Sq, Sk, hq, hkv, causal, sms);
}

static int flash_bwd_tc_impl(int kv_brows, const void* q, const void* k, const void* v, const void* o, const void* dout,
                               const void* lse, void* stats, void* dq_acc, void* dkv_acc, long long dkv_bytes, void* dq, void* dk, void* dv, int B, int Sq,
                               int Sk, int hq, int hkv, int d, long long q_ts, long long k_ts, long long v_ts,
                               long long o_ts, long long do_ts, long long dq_ts, long long dk_ts, long long dv_ts,
                               float scale, int causal, void* stream) {
  if (B <= 0 || Sq <= 0 || Sk <= 0 || hq % hkv) return LB_ERR_SHAPE;
  if ((q_ts | k_ts | v_ts | o_ts | do_ts | dq_ts | dk_ts | dv_ts) % 8) return LB_ERR_SHAPE;
  if (causal && Sk < Sq) return LB_ERR_SHAPE;
  if (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)dout | (uintptr_t)dq | (uintptr_t)dk | (uintptr_t)dv | (uintptr_t)o | (uintptr_t)stats | (uintptr_t)dq_acc) & 15)
    return LB_ERR_ARG;
  FaBwdParams p{(const bf16*)o, (const bf16*)dout, (const float*)lse, (float*)stats, (float*)dq_acc,
                (bf16*)dq, (bf16*)dk, (bf16*)dv, B, Sq, Sk, hq, hkv, o_ts, do_ts, dq_ts, dk_ts, dv_ts, scale, causal,
                kv_brows, 0, nullptr, nullptr, false};
  if (const int chunk = dkv_acc ? bwd_chunk(B, Sq, Sk, hq, hkv, causal, lb_num_sms()) : 0) {
    const long long bytes = bwd_parts_bytes(B, Sq, Sk, hq, hkv, d, causal, chunk);
    if (dkv_bytes >= 2 * bytes) {
      p.chunk = chunk;
      p.dk_acc = (float*)dkv_acc;
      p.dv_acc = p.dk_acc + bytes / (long long)sizeof(float);
    }
  }
  // Up to 128 keys a query block's dQ comes from one CTA, which writes it: no sums to clear, to add to and to convert.  Forward and backward, us, before / now,
  // d 64: B4 S128 12 heads inside its layer 58.5 / 57.0, B8 32 heads 29 / 25, B32 32q/8kv 66.6 / 55, B64 16 heads 97 / 83; B8 S100 16 heads d128 26 / 22.  (In
  // parts, which few CTAs with long loops get, dK and dV have to be converted all the same.)
  p.alone = Sk <= 128 && !p.chunk;
  cudaStream_t s = (cudaStream_t)stream;
  switch (d) {
    case 64: return launch_fa_bwd<64>(q, k, v, p, q_ts, k_ts, v_ts, s);
    case 128: return launch_fa_bwd<128>(q, k, v, p, q_ts, k_ts, v_ts, s);
    default: return LB_ERR_SHAPE;
  }
}

// Same contract as lb_flash_bwd (flash_attn.cu) except for the scratch: a workspace of ws_bytes >= lb_flash_bwd_ws_bytes(), 16-byte
// aligned, that need not be initialised (with the bytes of lb_flash_bwd_ws_bytes_kv() short launches are cut into more parts).  head_dim 64 or 128; causal needs Sk >= Sq.  K/V are the first Sk rows of every
// batch of a buffer with kv_brows rows per batch (the context-parallel gather buffers; Sk for plain tensors); dk / dv
// stay [B, Sk, hkv, d].
extern "C" int lb_flash_bwd_cp_ws(const void* q, const void* k, const void* v, const void* o, const void* dout,
                                  const void* lse, void* ws, long long ws_bytes, void* dq, void* dk, void* dv, int B, int Sq,
                                  int Sk, int kv_brows, int hq, int hkv, int d, long long q_ts, long long k_ts, long long v_ts,
                                  long long o_ts, long long do_ts, long long dq_ts, long long dk_ts, long long dv_ts,
                                  float scale, int causal, void* stream) {
  if (kv_brows < Sk) return LB_ERR_SHAPE;
  const long long need = lb_flash_bwd_ws_bytes(B, Sq, hq, d);
  if (!need) return LB_ERR_SHAPE;
  if (ws_bytes < need) return LB_ERR_CAPACITY;
  const long long n_pad = (long long)B * hq * ((Sq + 127) / 128) * 128;
  float* dkv_acc = ws_bytes > need ? (float*)ws + (2 + d) * n_pad : nullptr;
  return flash_bwd_tc_impl(kv_brows, q, k, v, o, dout, lse, ws, (float*)ws + 2 * n_pad, dkv_acc, ws_bytes - need, dq, dk, dv, B, Sq, Sk, hq, hkv, d,
                           q_ts, k_ts, v_ts, o_ts, do_ts, dq_ts, dk_ts, dv_ts, scale, causal, stream);
}

extern "C" int lb_flash_bwd_tc_ws(const void* q, const void* k, const void* v, const void* o, const void* dout,
                                  const void* lse, void* ws, long long ws_bytes, void* dq, void* dk, void* dv, int B, int Sq,
                                  int Sk, int hq, int hkv, int d, long long q_ts, long long k_ts, long long v_ts,
                                  long long o_ts, long long do_ts, long long dq_ts, long long dk_ts, long long dv_ts,
                                  float scale, int causal, void* stream) {
  return lb_flash_bwd_cp_ws(q, k, v, o, dout, lse, ws, ws_bytes, dq, dk, dv, B, Sq, Sk, Sk, hq, hkv, d, q_ts, k_ts, v_ts, o_ts,
                            do_ts, dq_ts, dk_ts, dv_ts, scale, causal, stream);
}

// The forms for callers that bring delta (fp32 [B, hq, Sq], not used) and dq_acc (fp32, B * hq * ceil(Sq/128) * 128 * d elements) as
// scratch: the row statistics need twice the padded rows, so they are allocated on the stream here.
extern "C" int lb_flash_bwd_cp(const void* q, const void* k, const void* v, const void* o, const void* dout,
                               const void* lse, void* delta, void* dq_acc, void* dq, void* dk, void* dv, int B, int Sq,
                               int Sk, int kv_brows, int hq, int hkv, int d, long long q_ts, long long k_ts,
                               long long v_ts, long long o_ts, long long do_ts, long long dq_ts, long long dk_ts,
                               long long dv_ts, float scale, int causal, void* stream) {
  (void)delta;
  if (kv_brows < Sk || !lb_flash_bwd_ws_bytes(B, Sq, hq, d)) return LB_ERR_SHAPE;
  void* stats = nullptr;
  cudaError_t e = cudaMallocAsync(&stats, (size_t)B * hq * ((Sq + 127) / 128) * 256 * sizeof(float), (cudaStream_t)stream);
  if (e != cudaSuccess) { cudaGetLastError(); g_lb_last_cuda_error = (int)e; return LB_ERR_LAUNCH; }
  const int rc = flash_bwd_tc_impl(kv_brows, q, k, v, o, dout, lse, stats, dq_acc, nullptr, 0, dq, dk, dv, B, Sq, Sk, hq, hkv, d, q_ts, k_ts,
                                   v_ts, o_ts, do_ts, dq_ts, dk_ts, dv_ts, scale, causal, stream);
  e = cudaFreeAsync(stats, (cudaStream_t)stream);
  if (rc == LB_OK && e != cudaSuccess) { g_lb_last_cuda_error = (int)e; return LB_ERR_LAUNCH; }
  return rc;
}

extern "C" int lb_flash_bwd_tc(const void* q, const void* k, const void* v, const void* o, const void* dout,
                               const void* lse, void* delta, void* dq_acc, void* dq, void* dk, void* dv, int B, int Sq,
                               int Sk, int hq, int hkv, int d, long long q_ts, long long k_ts, long long v_ts,
                               long long o_ts, long long do_ts, long long dq_ts, long long dk_ts, long long dv_ts,
                               float scale, int causal, void* stream) {
  return lb_flash_bwd_cp(q, k, v, o, dout, lse, delta, dq_acc, dq, dk, dv, B, Sq, Sk, Sk, hq, hkv, d, q_ts, k_ts, v_ts,
                         o_ts, do_ts, dq_ts, dk_ts, dv_ts, scale, causal, stream);
}
