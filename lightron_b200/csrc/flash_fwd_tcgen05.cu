// FlashAttention forward on the 5th-generation tensor cores (sm_100a), head_dim 64 or 128.
//
// A CTA works on one tile of 128 queries of one (batch, head) at a time; two CTAs share an SM.  Per 128-key block:
//     S = Q K^T          tcgen05.mma, 128x128xd, operands in 128B-swizzled smem (TMA), D in TMEM
//     softmax(S)         one thread per query row reads its row straight from TMEM
//                        (tcgen05.ld), so max / sum need no shuffles; P goes back to TMEM as
//                        packed bf16 pairs (tcgen05.st)
//     O (+)= P V         tcgen05.mma with the A operand in TMEM, 128 x d x 128, V is the MN-major
//                        B operand as it sits in memory; issued in two halves of 64 keys, the
//                        first while the exponentials of the second are still being computed
// P never touches shared memory, whose bandwidth (128 B/clk) the operand reads and the TMA writes share.
// O stays in TMEM for the whole key loop; when a row maximum grows the softmax threads rescale
// it in place (tcgen05.ld / st) before the next P V is issued.
// Warp roles (256 threads): warp 0 TMA producer, warp 1 MMA issuer and owner of the TMEM allocation, warps 2-3 idle, warps 4-7 softmax.
// What bounds it: 16 exponentials per clock per SM are 1024 cycles per 128x128 block against 542 (d = 64)
// or 1020 (d = 128) cycles of tensor pipe.  A tile's softmax, P V and next S follow one another, and the two CTAs of an SM fill each
// other's gaps: a block of a tile that has the SM to itself takes 2350 cycles (d = 64) / 3050 (d = 128), one of two tiles 3200 / 3700 on
// average.  At d = 128 the power limit comes on top (long loops run at 1.67 GHz).  Counters: exponentials 60 / 48 %, tensor pipe 30 / 48 % of the
// active cycles (B8 S2048 32q/4kv d64, B4 S2048 32q/8kv d128).  What the single cycles went into, and what each was worth:
//   * MMAs and loads are issued by an elected thread (elect_one has the cycles): with lane 0 in its place 242 us instead of 228 (B8 S2048
//     32q/4kv d64) and 557 instead of 488 (B1 S8192 32q/8kv d128);
//   * one CTA per tile instead of two tiles per CTA and CTAs that go on with the next tile (cluster launch control): prologue and
//     stores of a tile run under the other tile's blocks (d = 64 alone 265 -> 233 us);
//   * waits that are sure to succeed are put ahead of the one that is not (some 150 cycles each), O leaves through TMA stores.
// Loops of 0.35 s, two tiles per CTA / now, on one GPU: B8 S2048 32q/4kv d64 266 / 226 us, B1 S8192 32q/8kv d128 595 / 545,
// B3 S1531 32q/8kv d128 88 / 76, B1 S4096 8q/8kv d128 82 / 63.  Scaling and summing use two-wide fp32 instructions and the maximum
// three-input ones.  (Measured and not kept: a polynomial on the FMA pipe for one pair of exponentials in four; four tiles of 64-key blocks per
// SM at d = 64, 236 us, and two score buffers of 64 keys at d = 128, 753 us, which load each K and V byte in smaller boxes and
// leave one thread to issue everything; lists fixed in advance instead of launch control, 233 us against 224.)
// Layout / masking conventions are those of flash_attn.cu.
// All waits are bounded; on expiry a status word is set and the CTA drains and frees its TMEM.
#include <string.h>
#include "tcgen05.cuh"
#include "comm.cuh"

static __device__ unsigned int g_fa_status[4] = {0, 0, 0, 0};

namespace {
using namespace bw;

// Context-parallel extension ("all-gather KV inside the attention kernel"): the K/V operand is a
// gather buffer [B, S_full, hkv*d] in peer-visible memory that every rank of the CP group fills
// by PUSHING its own zig-zag chunks (rank r owns sequence chunks r and 2c-1-r) with coalesced
// peer stores from `n_mov` mover CTAs of this same kernel, counting each 128-key block in the
// destination's flag word.  The attention CTAs gate every 128-key block on its flag, so the
// exchange overlaps the softmax / MMA work on blocks that have already arrived.
constexpr int FA_MAX_RANKS = 8;
constexpr int FA_FWD_THREADS = 256;
// Registers per thread of the two warpgroups.  Two CTAs of 256 threads leave 128 per thread at launch; the issuing warpgroup gives most
// of its share to the softmax threads, of which each holds a row of 128 scores.  (Spills by -Xptxas -v: none at d = 64, 32 bytes
// stored and 36 loaded per thread at d = 128.)
constexpr int FA_REGS_ISSUE = 56, FA_REGS_SOFTMAX = 200;
static_assert(FA_REGS_ISSUE + FA_REGS_SOFTMAX <= 2 * 128, "a CTA has 256 x 128 registers");
struct FaPush {
  int n_mov, n_ranks, rank, chunk_rows, row_elems;   // row_elems = hkv * d
  const bf16 *k_src, *v_src;                         // this rank's [B, 2*chunk_rows, hkv, d], token strides below
  long long k_ts, v_ts;
  bf16* k_dst[FA_MAX_RANKS];                         // rank r's gather buffers [B, S_full, hkv*d]
  bf16* v_dst[FA_MAX_RANKS];
  unsigned int* flags[FA_MAX_RANKS];                 // rank r's block counters [B][S_full / 128]
};
// Division of 0 <= x < 2^31 by a divisor that is fixed for the launch: a multiplication by a rounded-up reciprocal (division by invariant
// integers, Granlund and Montgomery 1994; the host finds m, which is exact for such x).
struct FastDiv {
  unsigned int d, m, s;
  void set(unsigned int div) {
    d = div;
    s = 0;
    while (s < 31 && (1u << s) < div) s++;                                        // 2^(s-1) < d <= 2^s
    m = (unsigned int)((((unsigned long long)1 << (31 + s)) + div - 1) / div);    // < 2^32
  }
  __device__ __forceinline__ int div(int x) const { return (int)(((unsigned long long)(unsigned)x * m) >> (31 + s)); }
};

struct FaFwdParams {
  bf16* o;
  float* lse;
  int B, Sq, Sk, hq, hkv;
  long long o_ts;
  float scale;
  int causal;
  int kv_brows;                  // rows between consecutive batches in the K/V tensor maps (>= Sk)
  const unsigned int* kv_flags;  // null, or this rank's block counters [B][kv_brows / 128]
  unsigned int flag_target;
  int tiles_x;                   // query tiles (128 rows) per (batch, head)
  int steal;                     // CTAs go on with entries that have not been started
  int group;                     // (batch, head) pairs whose tiles are ordered together
  unsigned long long wait_ns;    // limit of a wait on a key block's arrival flag
  FastDiv by_grp, by_group, by_last, by_hq, by_rep;    // entries of a group, heads of a group / of the last one, hq, hq / hkv
};

// Three-input maximum; a NaN in any input is the result.
__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.NaN.ftz.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float max2(float a, float b) {
  float r;
  asm("max.NaN.ftz.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}

template <int D>
struct FaCfg {
  static constexpr int BM = 128, BN = 128;
  static constexpr int ATOMS = D / 64;
  static constexpr int SLOT_BYTES = 128 * 128;          // K: 128 keys x 64 columns; V: 128 keys x 64 columns or 64 keys x 128 columns
  static constexpr int SLOTS = 6 - ATOMS;               // 5 / 4
  static constexpr int UNITS = 2 * ATOMS;               // slots that a key block takes, K before V
  // TMEM columns: S fp32 [128], O fp32 [D], P packed bf16 [64], in the 256 that leave room for a second CTA.  With head_dim 64
  // P has columns of its own and S of the next key block is issued as soon as the softmax threads hold the current one in
  // registers.  With head_dim 128 P takes the first half of S's: the next S is then issued right behind P V (the tensor
  // pipe runs the two in order), and the other CTA's work fills the time of the softmax.
  static constexpr bool P_ALIAS = (D == 128);
  static constexpr int COL_S = 0, COL_O = 128, COL_P = P_ALIAS ? 0 : 192, TMEM_COLS = 256;
  static constexpr int OFF_Q = 0;
  static constexpr int OFF_RING = OFF_Q + ATOMS * SLOT_BYTES;
  static constexpr int OFF_OUT = OFF_RING + SLOTS * SLOT_BYTES;   // 64 columns of O on their way out, 4 KB per softmax warp
  static constexpr int OFF_BAR = OFF_OUT + SLOT_BYTES;
  static constexpr int NBAR = 2 + 2 * SLOTS + 9;
  static constexpr int SMEM = OFF_BAR + 256;
};
static_assert(FaCfg<64>::SMEM <= 115712 && FaCfg<128>::SMEM <= 115712, "two CTAs per SM");

template <int D>
__global__ void __launch_bounds__(FA_FWD_THREADS, 2)
fa_fwd_tc_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk,
                 const __grid_constant__ CUtensorMap tv, const __grid_constant__ CUtensorMap to, const FaFwdParams p,
                 const FaPush push) {
  using C = FaCfg<D>;
  if ((int)blockIdx.x < push.n_mov) {
    // ------------------------------- K/V mover CTAs -------------------------------
    // unit = (destination rank, batch, which of this rank's two chunks, 128-row block, K or V)
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    const int bpc = push.chunk_rows / 128;
    const int fpb = (2 * push.n_ranks * push.chunk_rows) / 128;       // flag words per batch
    const int units = push.n_ranks * p.B * 2 * bpc * 2;
    const int vec_per_row = push.row_elems / 8;
    for (int u = blockIdx.x; u < units; u += push.n_mov) {
      int t = u;
      const int kv = t & 1; t >>= 1;
      const int blk = t % bpc; t /= bpc;
      const int half = t & 1; t >>= 1;
      const int b = t % p.B; t /= p.B;
      const int dst = (push.rank + 1 + t) % push.n_ranks;
      const int chunk = half ? 2 * push.n_ranks - 1 - push.rank : push.rank;
      const long long lrow0 = (long long)b * 2 * push.chunk_rows + half * push.chunk_rows + blk * 128;
      const long long grow0 = (long long)b * fpb * 128 + (long long)chunk * push.chunk_rows + blk * 128;
      const bf16* src = kv ? push.v_src : push.k_src;
      const long long ts = kv ? push.v_ts : push.k_ts;
      bf16* dstp = (kv ? push.v_dst[dst] : push.k_dst[dst]) + grow0 * push.row_elems;
      // every warp copies its share of the block's rows, fences and counts by itself: while one warp
      // sits in its fence the others keep streaming
      for (int r = warp; r < 128; r += nwarps) {
        const uint4* sp = reinterpret_cast<const uint4*>(src + (lrow0 + r) * ts);
        uint4* dp = reinterpret_cast<uint4*>(dstp + (long long)r * push.row_elems);
        for (int v0 = 0; v0 < vec_per_row; v0 += 128) {
          uint4 a[4];
#pragma unroll
          for (int j = 0; j < 4; j++) if (v0 + j * 32 + lane < vec_per_row) a[j] = sp[v0 + j * 32 + lane];
#pragma unroll
          for (int j = 0; j < 4; j++) if (v0 + j * 32 + lane < vec_per_row) dp[v0 + j * 32 + lane] = a[j];
        }
      }
      __threadfence_system();
      __syncwarp();
      if (lane == 0)
        lbcomm::red_release_sys_add(push.flags[dst] + (grow0 >> 7), 1u);
    }
    return;
  }
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::OFF_BAR);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + C::NBAR + 5);     // behind two 16-byte answers
  int* s_abort = reinterpret_cast<int*>(tmem_slot + 1);     // {abort, extra wait in ms}: see bw::mbar_wait

  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;   // (uniform over the warp)
  const uint32_t sbase = smem_u32(smem);
  if (sbase & 1023u) {                                       // the swizzled tiles need it; nothing has been started yet
    if (threadIdx.x == 0) atomicExch(&g_fa_status[0], 4u);
    return;
  }
  const uint32_t bar0 = smem_u32(bars);
  // barrier map
  const uint32_t q_full = bar0, q_empty = bar0 + 8;
  auto full = [&](int s) { return bar0 + 8u * (2 + s); };
  auto empty = [&](int s) { return bar0 + 8u * (2 + C::SLOTS + s); };
  const uint32_t bar1 = bar0 + 8u * (2 + 2 * C::SLOTS);
  const uint32_t s_full = bar1, s_free = bar1 + 8, p_half = bar1 + 16, p_full = bar1 + 24, pv_done = bar1 + 32;   // p_half: P of 64 keys
  auto next_full = [&](int i) { return bar1 + 40u + 8u * i; };
  auto next_empty = [&](int i) { return bar1 + 56u + 8u * i; };
  const uint32_t next_slot = (bar0 + 8u * C::NBAR + 15u) & ~15u;

  // Grid: movers first (they must be resident before anything waits for data), then one entry per (batch, head, query tile).  Causal
  // tiles differ in length by up to the number of key blocks, so the longest tiles of all heads of a group come first and
  // the short ones fill the tail; a group is as many heads as keep their K / V in L2 together (launch_fa_fwd).  A resident CTA goes
  // on with entries that have not been started yet (cluster launch control: it cancels their launch and takes their place): the
  // loads and the first scores of a tile then run under the last softmax and the stores of the one before it, and no list is fixed in advance
  // (lists of equal length gave SMs that were done 12 % later than the mean).
  volatile int* abort_flag = s_abort;
  const int off = p.Sk - p.Sq;
  struct Tile { int m0, b, h, hk, nb; };
  auto tile_of = [&](int cta) {
    Tile t;
    const int cid = cta - push.n_mov;
    const int grp = p.by_grp.div(cid);
    const int in_grp = cid - grp * (int)p.by_grp.d;
    const FastDiv& heads = (grp + 1) * p.group <= p.hq * p.B ? p.by_group : p.by_last;
    const int row = heads.div(in_grp);
    const int bh = grp * p.group + in_grp - row * (int)heads.d;
    t.m0 = (p.tiles_x - 1 - row) * C::BM;
    t.b = p.by_hq.div(bh);
    t.h = bh - t.b * p.hq;
    t.hk = p.by_rep.div(t.h);
    t.nb = (p.Sk + C::BN - 1) / C::BN;
    if (p.causal) t.nb = min(t.nb, (t.m0 + C::BM - 1 + off) / C::BN + 1);
    return t;
  };
  // Entry n + 1 of this CTA: the answer to request n, or -1 at the end.
  auto next_cta = [&](int n) -> int {
    if (!p.steal || !mbar_wait(next_full(n & 1), (uint32_t)(n >> 1) & 1u, abort_flag)) return -1;
    const int cta = cancel_result(next_slot + 16u * (n & 1));
    fence_proxy_async_smem();
    return cta;
  };

  if (threadIdx.x == 0) {
    s_abort[0] = 0;
    s_abort[1] = p.kv_flags ? wait_extra_ms(p.wait_ns) : 0;
    mbar_init(q_full, 1);
    mbar_init(q_empty, 1);
    for (int s = 0; s < C::SLOTS; s++) { mbar_init(full(s), 1); mbar_init(empty(s), 1); }
    mbar_init(s_full, 1);
    mbar_init(pv_done, 1);
    mbar_init(s_free, 4);
    mbar_init(p_half, 4);
    mbar_init(p_full, 4);
    for (int i = 0; i < 2; i++) { mbar_init(next_full(i), 1); mbar_init(next_empty(i), 5); }   // the issuer and four softmax warps read
    mbar_init_fence();
    prefetch_tmap(&tq); prefetch_tmap(&tk); prefetch_tmap(&tv); prefetch_tmap(&to);
  }
  if (warp == 1) tmem_alloc(smem_u32(tmem_slot), C::TMEM_COLS);
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  if (!p.steal && !push.n_mov && !p.kv_flags) grid_go();
  grid_wait();

  if (warp < 4) {
    reg_dec<FA_REGS_ISSUE>();
    if (warp == 0) {
      // ------------------------------- TMA producer -------------------------------
      if (elect_one()) {
        bool ok = true;
        int slot = 0;
        uint32_t phase = 0;
        int asked = 0;
        for (int n = 0, cta = (int)blockIdx.x; ok && cta >= 0; n++) {
          if (p.steal) {
            if (!mbar_wait(next_empty(n & 1), ((uint32_t)(n >> 1) & 1u) ^ 1u, abort_flag)) { ok = false; break; }
            mbar_expect_tx(next_full(n & 1), 16);
            cancel_next(next_slot + 16u * (n & 1), next_full(n & 1));
            asked = n + 1;
          }
          const Tile t = tile_of(cta);
          if (!mbar_wait(q_empty, (uint32_t)(n & 1) ^ 1u, abort_flag)) { ok = false; break; }
          mbar_expect_tx(q_full, C::ATOMS * C::SLOT_BYTES);
#pragma unroll
          for (int a = 0; a < C::ATOMS; a++)
            tma_load_2d(sbase + C::OFF_Q + a * C::SLOT_BYTES, &tq, t.h * D + a * 64, t.b * p.Sq + t.m0, q_full);
          for (int j = 0; j < t.nb && ok; j++) {
            if (p.kv_flags) {
              // this 128-key block is pushed by its owner: wait for its counter, then order the
              // peer's generic-proxy writes before the TMA (async proxy) reads
              if (!lbcomm::flag_wait_ge(p.kv_flags + (long long)t.b * (p.kv_brows >> 7) + j, p.flag_target, p.wait_ns)) { *abort_flag = 1; ok = false; break; }
              asm volatile("fence.proxy.async;" ::: "memory");
            }
            const int key0 = j * C::BN;
#pragma unroll
            for (int u = 0; u < C::UNITS; u++) {
              if (ok && !mbar_wait(empty(slot), phase ^ 1u, abort_flag)) ok = false;
              if (!ok) break;
              const uint32_t dst = sbase + C::OFF_RING + slot * C::SLOT_BYTES, bar = full(slot);
              mbar_expect_tx(bar, C::SLOT_BYTES);
              if (u < C::ATOMS) {
                tma_load_2d(dst, &tk, t.hk * D + u * 64, t.b * p.kv_brows + key0, bar);               // box 128 keys x 64 columns
              } else {
                const int half = u - C::ATOMS;                                    // head_dim 128: keys 0-63, then 64-127
#pragma unroll
                for (int a = 0; a < 2; a++)                                       // boxes 64 keys x 64 columns
                  tma_load_3d(dst + a * 8192, &tv, t.hk * D + (D == 128 ? a * 64 : 0), key0 + (D == 128 ? half * 64 : a * 64), t.b, bar);
              }
              if (++slot == C::SLOTS) { slot = 0; phase ^= 1u; }
            }
          }
          if (ok) cta = next_cta(n);
        }
        if (!ok) {
          atomicExch(&g_fa_status[0], 1u);
          if (asked) mbar_wait(next_full((asked - 1) & 1), (uint32_t)((asked - 1) >> 1) & 1u, abort_flag);   // nothing arrives after the CTA's end
        }
      }
    } else if (warp == 1) {
      // ------------------------------- MMA issuer -------------------------------
      // Blocking waits in a fixed order.  Per tile S(0); then per key block, head_dim 64: S(j+1) as soon as the softmax threads hold S(j) in
      // registers, and P(j) V in two halves as P(j) arrives; head_dim 128: P(j) V, then S(j+1) into the columns that P(j) leaves.
      if (elect_one()) {
        const uint32_t idesc_s = make_idesc(C::BM, C::BN, 0, 0);
        const uint32_t idesc_o = make_idesc(C::BM, D, 0, 1);
        // descriptor bases; a slot / k-step only changes the 16-byte-granular start address
        const uint64_t qa = make_desc(sbase + C::OFF_Q, 16, 1024);
        const uint64_t dk0 = make_desc(sbase + C::OFF_RING, 16, 1024);
        const uint64_t dv0 = make_desc(sbase + C::OFF_RING, 8192, 1024);
        const uint32_t s_dst = tmem_base + C::COL_S;
        const uint32_t o_dst = tmem_base + C::COL_O;
        const uint32_t pa = tmem_base + C::COL_P;          // 8 columns per K = 16 slice
        bool ok = true;
        // slots are taken in load order: K (ATOMS slots), then V of every block; head_dim 64 takes K of the next block before V of the current
        auto ring = [&](int& slot, uint32_t& phase, int step) { slot += step; if (slot >= C::SLOTS) { slot -= C::SLOTS; phase ^= 1u; } };
        int ks = 0, vs = C::ATOMS;                      // next slot of K and of V, and their phases
        uint32_t kp = 0, vp = 0;
        uint32_t g = 0;                                 // key blocks so far, over all tiles: the phase of the per-block barriers
        auto k_ready = [&]() -> bool {                  // the next block's K has arrived
          if (!mbar_wait(full(ks), kp, abort_flag)) return false;
          if (C::ATOMS == 1) return true;
          const bool wrap = ks + 1 == C::SLOTS;
          return mbar_wait(full(wrap ? 0 : ks + 1), wrap ? kp ^ 1u : kp, abort_flag);
        };
        auto issue_s = [&](bool last) {                 // S = Q K^T of the next block (K is there), then release its slots of K (and Q)
          fence_after();
#pragma unroll
          for (int a = 0; a < C::ATOMS; a++) {
            const uint64_t ka = dk0 + (uint64_t)((ks * C::SLOT_BYTES) >> 4);
#pragma unroll
            for (int s = 0; s < 4; s++)
              umma_bf16(s_dst, qa + (uint64_t)((a * C::SLOT_BYTES + s * 32) >> 4), ka + (uint64_t)((s * 32) >> 4), idesc_s, (a | s) ? 1u : 0u);
            if (a == C::ATOMS - 1) umma_commit(s_full);
            umma_commit(empty(ks));
            ring(ks, kp, a == C::ATOMS - 1 ? C::UNITS - C::ATOMS + 1 : 1);
          }
          if (last) umma_commit(q_empty);
        };
        // O += P V of block g, then release its slots of V.  What a step waits for is waited for ahead of the wait for P, which is
        // the last to come: a wait takes some 150 cycles even where there is nothing to wait for.
        auto issue_pv = [&](bool first, bool last) -> bool {
#pragma unroll
          for (int half = 0; half < 2; half++) {
            if ((D == 128 || half == 0) && !mbar_wait(full(vs), vp, abort_flag)) return false;
            if (half == 1 && C::P_ALIAS && !last && !k_ready()) return false;
            if (!mbar_wait(half ? p_full : p_half, g & 1u, abort_flag)) return false;
            fence_after();
            const uint64_t va = dv0 + (uint64_t)((vs * C::SLOT_BYTES + (D == 128 ? 0 : half * 8192)) >> 4);
#pragma unroll
            for (int s = 0; s < 4; s++)
              umma_bf16_ta(o_dst, pa + 8u * (half * 4 + s), va + (uint64_t)((s * 2048) >> 4), idesc_o, (half | s) ? 1u : (first ? 0u : 1u));
            if (half && (!C::P_ALIAS || last)) umma_commit(pv_done);
            if (D == 128 || half) {
              umma_commit(empty(vs));
              ring(vs, vp, half ? C::ATOMS + 1 : 1);
            }
          }
          return true;
        };
        for (int n = 0, cta = (int)blockIdx.x; ok && cta >= 0; n++) {
          const Tile t = tile_of(cta);
          ok = k_ready() && mbar_wait(q_full, (uint32_t)n & 1u, abort_flag);
          if (ok && !C::P_ALIAS && n > 0) ok = mbar_wait(s_free, (g - 1) & 1u, abort_flag);
          if (ok) issue_s(t.nb == 1);
          for (int j = 0; j < t.nb && ok; j++, g++) {
            const bool last = j + 1 == t.nb;
            if (!C::P_ALIAS && !last) {
              ok = k_ready() && mbar_wait(s_free, g & 1u, abort_flag);
              if (ok) issue_s(j + 2 == t.nb);
            }
            if (ok) ok = issue_pv(j == 0, last);
            if (C::P_ALIAS && ok && !last) issue_s(j + 2 == t.nb);
          }
          if (!ok) break;
          cta = next_cta(n);
          if (cta >= 0) mbar_arrive(next_empty(n & 1));
        }
        if (!ok) atomicExch(&g_fa_status[0], 2u);
      }
    }
  } else {
    // ------------------------------- softmax warps -------------------------------
    reg_inc<FA_REGS_SOFTMAX>();
    const int quad = warp & 3;
    const uint32_t lane_addr = tmem_base + ((uint32_t)(quad * 32) << 16);
    const uint32_t ts_addr = lane_addr + C::COL_S;
    const uint32_t to_addr = lane_addr + C::COL_O;
    const uint32_t tp_addr = lane_addr + C::COL_P;
    const float sl2 = p.scale * 1.4426950408889634f;
    const f32x2 sl2x2 = pack2(sl2, sl2);
    bool ok = true;
    auto arrive = [&](uint32_t bar) {              // once per warp
      fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar);
    };
    uint32_t g = 0;                                // key blocks so far, over all tiles
    bool s_ready = false;                          // S of the next block was seen complete
    for (int n = 0, cta = (int)blockIdx.x; ok && cta >= 0; n++) {
      const Tile t = tile_of(cta);
      const int m0 = t.m0, nb = t.nb;
      const int row = m0 + quad * 32 + lane;         // query index inside the sequence
      float m_i = -INFINITY, m_s = 0.f, l_i = 0.f;
      for (int j = 0; j < nb; j++, g++) {
        if (!s_ready && !mbar_wait(s_full, g & 1u, abort_flag)) { ok = false; break; }
        fence_after();
        uint32_t r[128];
        const int c0 = j * C::BN;
        const int warp_row0 = m0 + quad * 32;
        const bool need_mask = (c0 + C::BN > p.Sk) || (p.causal && (c0 + C::BN - 1 > warp_row0 + off));
        const int lim = (p.causal ? min(p.Sk - 1, row + off) : p.Sk - 1) - c0;   // last visible column of this block
        auto mask = [&](int i0) {
          if (need_mask) {
#pragma unroll
            for (int i = i0; i < i0 + 64; i++)
              if (i > lim) r[i] = 0xff800000u;           // -inf
          }
        };
        // exponentials of 64 columns, packed as bf16 pairs (column c of P holds keys 2c, 2c+1)
        auto exps = [&](int i0, uint32_t* pr, f32x2* rs2) {
          const f32x2 nms2 = pack2(-m_s, -m_s);
          rs2[0] = rs2[1] = pack2(0.f, 0.f);
#pragma unroll
          for (int c = 0; c < 32; c++) {
            const int i = i0 + c * 2;
            float e0, e1;
            unpack2(fma2(pack2(__uint_as_float(r[i]), __uint_as_float(r[i + 1])), sl2x2, nms2), e0, e1);
            e0 = exp2f(e0);
            e1 = exp2f(e1);
            rs2[c & 1] = add2(rs2[c & 1], pack2(e0, e1));
            bf162 pk = __floats2bfloat162_rn(e0, e1);
            pr[c] = *reinterpret_cast<uint32_t*>(&pk);
          }
        };
        auto row_max = [&]() {                           // four independent chains
          float mx4[4] = {m_i, m_i, m_i, m_i};
#pragma unroll
          for (int i = 0; i < 128; i += 2) mx4[(i >> 1) & 3] = max3(mx4[(i >> 1) & 3], __uint_as_float(r[i]), __uint_as_float(r[i + 1]));
          return max2(max2(mx4[0], mx4[1]), max2(mx4[2], mx4[3]));
        };
        tmem_ld32(ts_addr, r);
        tmem_ld32(ts_addr + 32, r + 32);
        tmem_ld32(ts_addr + 64, r + 64);
        tmem_ld32(ts_addr + 96, r + 96);
        tmem_ld_wait();
        if (!C::P_ALIAS) arrive(s_free);                 // S may be overwritten by the next key block
        mask(0);
        mask(64);
        // Lazy reference maximum: the old one stays unless the new maximum is more than 2^8 above it, so that O and l rarely
        // need rescaling (values stay below 2^8 relative to it).  So the first 64 exponentials are computed with the old one, while the
        // maximum that tells whether it may stay is still being found, and once more in the rare block where it may not.
        uint32_t pr[32];
        f32x2 rs2[2], rt2[2];
        const bool pv_ready = !C::P_ALIAS && j > 0 && mbar_test_wait(pv_done, (g - 1) & 1u);   // asked ahead of its use
        if (j > 0) exps(0, pr, rs2);
        float m_new = row_max();
        const bool grow = !(m_i != -INFINITY && (m_new - m_i) * sl2 <= 8.f);
        const bool any_grow = __any_sync(0xffffffffu, grow);
        float corr = 1.f;
        if (any_grow) {
          if (!grow) m_new = m_i;
          // (a row with a score of +inf has no softmax: NaN, as inf - inf gives)
          m_s = (m_new == -INFINITY) ? 0.f : (m_new == INFINITY ? __int_as_float(0x7fffffff) : m_new * sl2);
          corr = (m_i == -INFINITY) ? 0.f : exp2f(m_i * sl2 - m_s);
          l_i *= corr;
          m_i = m_new;
          exps(0, pr, rs2);
        }
        if (j > 0) {
          // previous P V finished: O is stable and the P columns may be overwritten.  (head_dim 128: S(j) was
          // issued behind it by the same thread, so its completion says that P V has completed too.)
          if (!C::P_ALIAS) {
            if (!pv_ready && !mbar_wait(pv_done, (g - 1) & 1u, abort_flag)) { ok = false; break; }
            fence_after();
          }
          if (any_grow) {
#pragma unroll 1
            for (int c = 0; c < D / 32; c++) {
              uint32_t o[32];
              tmem_ld32(to_addr + c * 32, o);
              tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 32; i++) o[i] = __float_as_uint(__uint_as_float(o[i]) * corr);
              tmem_st32(to_addr + c * 32, o);
            }
            tmem_st_wait();
          }
        }
        // P goes back to TMEM, the first half in flight while the second is computed
        tmem_st32(tp_addr, pr);
        tmem_st_wait();
        arrive(p_half);
        s_ready = !C::P_ALIAS && j + 1 < nb && mbar_test_wait(s_full, (g + 1) & 1u);
        exps(64, pr, rt2);
        tmem_st32(tp_addr + 32, pr);
        tmem_st_wait();
        arrive(p_full);
        rs2[0] = add2(rs2[0], rt2[0]);
        rs2[1] = add2(rs2[1], rt2[1]);
        float rs[4];
        unpack2(rs2[0], rs[0], rs[1]);
        unpack2(rs2[1], rs[2], rs[3]);
        l_i += (rs[0] + rs[1]) + (rs[2] + rs[3]);
      }
      if (ok) {
        cta = next_cta(n);
        __syncwarp();
        if (lane == 0 && cta >= 0) mbar_arrive(next_empty(n & 1));
      }
      if (ok && !mbar_wait(pv_done, C::P_ALIAS ? (uint32_t)n & 1u : (g - 1) & 1u, abort_flag)) ok = false;
      if (!ok) break;
      fence_after();
      const float inv = l_i > 0.f ? 1.f / l_i : 0.f;
      // 64 columns at a time through shared memory: a row per lane stored straight to memory is 32 separate lines for every 16 bytes
      // per lane, which kept the load/store unit busy for as long as one and a half key blocks take
      uint8_t* out = smem + C::OFF_OUT + quad * 4096;
#pragma unroll
      for (int c = 0; c < D / 64; c++) {
        uint32_t r[64];
        tmem_ld32(to_addr + c * 64, r);
        tmem_ld32(to_addr + c * 64 + 32, r + 32);
        tmem_ld_wait();
        if (lane == 0) bulk_wait_read_but<0>();
        __syncwarp();
#pragma unroll
        for (int g8 = 0; g8 < 8; g8++) {
          float f[8];
#pragma unroll
          for (int i = 0; i < 8; i++) f[i] = __uint_as_float(r[g8 * 8 + i]) * inv;
          *reinterpret_cast<uint4*>(out + sw128_off(lane, g8)) = pack8(f);
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0 && m0 + quad * 32 < p.Sq) {
          tma_store_3d(&to, smem_u32(out), t.h * D + c * 64, m0 + quad * 32, t.b);
          bulk_commit();
        }
      }
      if (row < p.Sq)
        p.lse[((long long)t.b * p.hq + t.h) * p.Sq + row] = (l_i > 0.f) ? m_i * p.scale + logf(l_i) : -INFINITY;
    }
    if (lane == 0) bulk_wait_read_but<0>();        // nothing reads shared memory after the CTA's end
    if (!ok && lane == 0) atomicExch(&g_fa_status[0], 3u);
  }

  fence_before();
  __syncthreads();
  if (warp == 1) {
    fence_after();
    tmem_dealloc(tmem_base, C::TMEM_COLS);
  }
}

// One key block (Sk <= 128) and no more tiles than run at a time: a launch is then one chain from the loads to the stores, and what it takes is the instructions
// of a softmax warp, straight-line code for its columns that mostly comes from L2.  So a row is two threads', 64 keys each, in eight warps: maxima and sums meet in
// shared memory, P takes the columns of S.  The products, the exponentials and the order of the sums are those of fa_fwd_tc_kernel: the results are the same
// bits.  fa_fwd_tc_kernel / this, us, as graphs: 12 layers of 128 tokens, 12 heads of 64, 455 / 411; forward and backward of 4 x 128 tokens, 12 heads of 64 15.6 / 14.4, of
// 8 x 100, 16 heads of 128 20.5 / 18.5; the layer around the former 54.7 / 52.6.  With more tiles than run at a time the other kernel's loads and scores of a tile under
// the last one's softmax count for more (forward alone, d 64: 256 tiles -> 5.4 here, 320 8.3 / 8.7, 1024 14.6 / 18.1, 4096 47 / 74; d 128, 512 tiles 12.1 / 15.0).
constexpr int FA_ONE_THREADS = 320;
__device__ __forceinline__ void named_sync(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }
template <int D>
struct FaOneCfg {
  static constexpr int ATOMS = D / 64, SLOT_BYTES = 128 * 128;
  static constexpr int COL_S = 0, COL_P = 0, COL_O = 128, TMEM_COLS = 256;
  static constexpr int OFF_Q = 0, OFF_K = ATOMS * SLOT_BYTES, OFF_V = 2 * ATOMS * SLOT_BYTES;
  static constexpr int OFF_MAX = 3 * ATOMS * SLOT_BYTES;        // [2][128] maxima, then [2][128] x 4 sums
  static constexpr int OFF_SUM = OFF_MAX + 2 * 128 * 4, OFF_BAR = OFF_SUM + 2 * 128 * 16;
  static constexpr int SMEM = OFF_BAR + 64;
};
static_assert(FaOneCfg<128>::SMEM <= 115712, "two CTAs per SM");

template <int D>
__global__ void __launch_bounds__(FA_ONE_THREADS, 2)
fa_fwd_one_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk, const __grid_constant__ CUtensorMap tv, const FaFwdParams p) {
  using C = FaOneCfg<D>;
  extern __shared__ __align__(1024) uint8_t smem[];
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;   // (uniform over the warp)
  const uint32_t sbase = smem_u32(smem);
  if (sbase & 1023u) {                                       // the swizzled tiles need it; nothing has been started yet
    if (threadIdx.x == 0) atomicExch(&g_fa_status[0], 4u);
    return;
  }
  const uint32_t qk_full = sbase + C::OFF_BAR, v_full = qk_full + 8, s_full = qk_full + 16, p_full = qk_full + 24, o_full = qk_full + 32;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + C::OFF_BAR + 40);
  int* s_abort = reinterpret_cast<int*>(tmem_slot + 1);      // {abort, extra wait in ms}: see bw::mbar_wait
  volatile int* abort_flag = s_abort;
  const int m0 = (int)blockIdx.y * 128, bh = (int)blockIdx.x;
  const int b = p.by_hq.div(bh), h = bh - b * p.hq, hk = p.by_rep.div(h);
  if (threadIdx.x == 0) {
    s_abort[0] = s_abort[1] = 0;
    mbar_init(qk_full, 1);
    mbar_init(v_full, 1);
    mbar_init(s_full, 1);
    mbar_init(p_full, 8);
    mbar_init(o_full, 1);
    mbar_init_fence();
    prefetch_tmap(&tq); prefetch_tmap(&tk); prefetch_tmap(&tv);
  }
  if (warp == 1) tmem_alloc(smem_u32(tmem_slot), C::TMEM_COLS);
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  grid_go();
  grid_wait();

  if (warp == 0) {
    if (elect_one()) {
      mbar_expect_tx(qk_full, 2 * C::ATOMS * C::SLOT_BYTES);
#pragma unroll
      for (int a = 0; a < C::ATOMS; a++) {
        tma_load_2d(sbase + C::OFF_Q + a * C::SLOT_BYTES, &tq, h * D + a * 64, b * p.Sq + m0, qk_full);
        tma_load_2d(sbase + C::OFF_K + a * C::SLOT_BYTES, &tk, hk * D + a * 64, b * p.kv_brows, qk_full);
      }
      mbar_expect_tx(v_full, C::ATOMS * C::SLOT_BYTES);
#pragma unroll
      for (int half = 0; half < 2; half++)
#pragma unroll
        for (int a = 0; a < C::ATOMS; a++)                   // boxes 64 keys x 64 columns
          tma_load_3d(sbase + C::OFF_V + (half * C::ATOMS + a) * 8192, &tv, hk * D + a * 64, half * 64, b, v_full);
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t idesc_s = make_idesc(128, 128, 0, 0), idesc_o = make_idesc(128, D, 0, 1);
      const uint64_t qa = make_desc(sbase + C::OFF_Q, 16, 1024), ka = make_desc(sbase + C::OFF_K, 16, 1024), va = make_desc(sbase + C::OFF_V, 8192, 1024);
      bool ok = mbar_wait(qk_full, 0, abort_flag);
      if (ok) {
        fence_after();
#pragma unroll
        for (int i = 0; i < D / 16; i++) {
          const uint64_t at = (uint64_t)(((i >> 2) * C::SLOT_BYTES + (i & 3) * 32) >> 4);
          umma_bf16(tmem_base + C::COL_S, qa + at, ka + at, idesc_s, i ? 1u : 0u);
        }
        umma_commit(s_full);
        ok = mbar_wait(v_full, 0, abort_flag) && mbar_wait(p_full, 0, abort_flag);
      }
      if (ok) {
        fence_after();
#pragma unroll
        for (int i = 0; i < 8; i++)
          umma_bf16_ta(tmem_base + C::COL_O, tmem_base + C::COL_P + 8u * i, va + (uint64_t)(((i >> 2) * C::ATOMS * 8192 + (i & 3) * 2048) >> 4), idesc_o, i ? 1u : 0u);
        umma_commit(o_full);
      } else {
        atomicExch(&g_fa_status[0], 2u);
      }
    }
  } else {
    const int set = warp >= 6 ? 1 : 0, quad = warp & 3;
    const int rit = quad * 32 + lane, row = m0 + rit;        // query row in the tile, and in the sequence
    const uint32_t lane_addr = tmem_base + ((uint32_t)(quad * 32) << 16);
    float* mx = reinterpret_cast<float*>(smem + C::OFF_MAX);
    float4* sums = reinterpret_cast<float4*>(smem + C::OFF_SUM);
    const float sl2 = p.scale * 1.4426950408889634f;
    const f32x2 sl2x2 = pack2(sl2, sl2);
    const int c0 = set * 64;
    const int lim = (p.causal ? min(p.Sk - 1, row + p.Sk - p.Sq) : p.Sk - 1) - c0;   // last visible column
    uint32_t r[64];
    bool ok = __all_sync(0xffffffffu, mbar_wait(s_full, 0, abort_flag));
    float m = -INFINITY;
    if (ok) {
      fence_after();
      tmem_ld32(lane_addr + C::COL_S + c0, r);
      tmem_ld32(lane_addr + C::COL_S + c0 + 32, r + 32);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 64; i++)
        if (i > lim) r[i] = 0xff800000u;                     // -inf
      float mx4[4] = {m, m, m, m};
#pragma unroll
      for (int i = 0; i < 64; i += 2) mx4[(i >> 1) & 3] = max3(mx4[(i >> 1) & 3], __uint_as_float(r[i]), __uint_as_float(r[i + 1]));
      m = max2(max2(mx4[0], mx4[1]), max2(mx4[2], mx4[3]));
    }
    mx[set * 128 + rit] = m;
    fence_before();
    named_sync(1, 256);                                      // (whether or not the wait ended well; S has been read)
    fence_after();
    m = max2(mx[rit], mx[128 + rit]);
    // (a row with a score of +inf has no softmax: NaN, as inf - inf gives)
    const float m_s = m == -INFINITY ? 0.f : (m == INFINITY ? __int_as_float(0x7fffffff) : m * sl2);
    if (ok) {
      const f32x2 nms2 = pack2(-m_s, -m_s);
      f32x2 rs2[2] = {pack2(0.f, 0.f), pack2(0.f, 0.f)};
      uint32_t pr[32];
#pragma unroll
      for (int c = 0; c < 32; c++) {
        float e0, e1;
        unpack2(fma2(pack2(__uint_as_float(r[2 * c]), __uint_as_float(r[2 * c + 1])), sl2x2, nms2), e0, e1);
        e0 = exp2f(e0);
        e1 = exp2f(e1);
        rs2[c & 1] = add2(rs2[c & 1], pack2(e0, e1));
        bf162 pk = __floats2bfloat162_rn(e0, e1);
        pr[c] = *reinterpret_cast<uint32_t*>(&pk);
      }
      tmem_st32(lane_addr + C::COL_P + set * 32, pr);
      tmem_st_wait();
      float4 s4;
      unpack2(rs2[0], s4.x, s4.y);
      unpack2(rs2[1], s4.z, s4.w);
      sums[set * 128 + rit] = s4;
      fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full);
    }
    named_sync(1, 256);
    const float4 x = sums[rit], y = sums[128 + rit];
    const float l = (x.x + y.x + (x.y + y.y)) + (x.z + y.z + (x.w + y.w));
    ok = ok && mbar_wait(o_full, 0, abort_flag);
    ok = __all_sync(0xffffffffu, ok);
    if (ok) {
      fence_after();
      const float inv = l > 0.f ? 1.f / l : 0.f;
      uint32_t o[D / 2];
#pragma unroll
      for (int c = 0; c < D / 64; c++) tmem_ld32(lane_addr + C::COL_O + set * (D / 2) + c * 32, o + c * 32);
      tmem_ld_wait();
      if (row < p.Sq) {
        bf16* out = p.o + ((long long)b * p.Sq + row) * p.o_ts + (long long)h * D + set * (D / 2);
#pragma unroll
        for (int g = 0; g < D / 16; g++) {
          float f[8];
#pragma unroll
          for (int i = 0; i < 8; i++) f[i] = __uint_as_float(o[g * 8 + i]) * inv;
          *reinterpret_cast<uint4*>(out + g * 8) = pack8(f);
        }
        if (set == 0) p.lse[((long long)b * p.hq + h) * p.Sq + row] = l > 0.f ? m * p.scale + logf(l) : -INFINITY;
      }
    } else if (lane == 0) {
      atomicExch(&g_fa_status[0], 3u);
    }
  }

  fence_before();
  __syncthreads();
  if (warp == 1) {
    fence_after();
    tmem_dealloc(tmem_base, C::TMEM_COLS);
  }
}

template <int D>
int launch_fa_fwd(const void* q, const void* k, const void* v, FaFwdParams p, const FaPush& push, long long q_ts,
                  long long k_ts, long long v_ts, cudaStream_t s) {
  using C = FaCfg<D>;
  CUtensorMap tq, tk, tv, to;
  int rc;
  const uint64_t kv_rows = (uint64_t)(p.B - 1) * p.kv_brows + p.Sk;
  if ((rc = make_map_bf16(&tq, q, (uint64_t)p.hq * D, (uint64_t)p.B * p.Sq, (uint64_t)q_ts, 64, 128))) return rc;
  if ((rc = make_map_bf16(&tk, k, (uint64_t)p.hkv * D, kv_rows, (uint64_t)k_ts, 64, 128))) return rc;
  // (keys past a sequence's last have weights of zero, but zero times the infinity or NaN of the next sequence's V is NaN: they are loaded as zeros)
  if ((rc = make_map_bf16_3d(&tv, v, (uint64_t)p.hkv * D, (uint64_t)p.Sk, (uint64_t)p.kv_brows, (uint64_t)p.B, (uint64_t)v_ts, 64, 64))) return rc;
  if ((rc = make_map_bf16_3d(&to, p.o, (uint64_t)p.hq * D, (uint64_t)p.Sq, (uint64_t)p.Sq, (uint64_t)p.B, (uint64_t)p.o_ts, 64, 32))) return rc;
  static bool attr = false;
  if (!attr) {
    // the register split must fit in what the launch allocates, or it would wait for registers that nobody gives back
    cudaFuncAttributes fa;
    if (cudaFuncGetAttributes(&fa, fa_fwd_tc_kernel<D>) != cudaSuccess || (fa.numRegs + 7) / 8 * 8 * 2 < FA_REGS_ISSUE + FA_REGS_SOFTMAX) return LB_ERR_LAUNCH;
    cudaFuncSetAttribute(fa_fwd_tc_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
    cudaFuncSetAttribute(fa_fwd_one_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, FaOneCfg<D>::SMEM);
    attr = true;
  }
  p.tiles_x = (p.Sq + 127) / 128;
  // heads ordered together: as many as have their K / V in 48 MB (of 126 MB of L2), whole GQA groups
  const long long kv_bytes = 4LL * D * p.Sk;
  const long long kv_heads = kv_bytes >= (48LL << 20) ? 1 : (48LL << 20) / kv_bytes;
  p.group = (int)(kv_heads * (p.hq / p.hkv) < (long long)p.hq * p.B ? kv_heads * (p.hq / p.hkv) : (long long)p.hq * p.B);
  p.wait_ns = g_lb_flag_wait_ns;
  const long long grid = (long long)push.n_mov + (long long)p.tiles_x * p.hq * p.B;
  if (grid > 2147483647LL) return LB_ERR_SHAPE;
  p.by_grp.set((unsigned)(p.tiles_x * p.group));
  p.by_group.set((unsigned)p.group);
  p.by_last.set((unsigned)(p.hq * p.B % p.group ? p.hq * p.B % p.group : p.group));
  p.by_hq.set((unsigned)p.hq);
  p.by_rep.set((unsigned)(p.hq / p.hkv));
  // (a mover's place is not to be taken; with all tiles resident at once there is none to take)
  p.steal = push.n_mov == 0 && grid > 2 * lb_num_sms();
  if (p.Sk <= 128 && push.n_mov == 0 && !p.kv_flags && !p.steal)
    return lb_launch_cluster(true, 1, fa_fwd_one_kernel<D>, dim3((unsigned)(p.hq * p.B), (unsigned)p.tiles_x), FA_ONE_THREADS, FaOneCfg<D>::SMEM, s, tq, tk, tv, p);
  return lb_launch_cluster(push.n_mov == 0 && !p.kv_flags, 1, fa_fwd_tc_kernel<D>, (unsigned)grid, FA_FWD_THREADS, C::SMEM, s, tq, tk, tv, to, p, push);
}

}  // namespace

// Copies the status words of the tcgen05 attention kernels to host memory and clears them.
extern "C" int lb_flash_status(void* out) {
  cudaError_t e = cudaMemcpyFromSymbol(out, g_fa_status, sizeof(unsigned int) * 4);
  if (e != cudaSuccess) { g_lb_last_cuda_error = (int)e; return LB_ERR_LAUNCH; }
  unsigned int zeros[4] = {0, 0, 0, 0};
  cudaMemcpyToSymbol(g_fa_status, zeros, sizeof(zeros));
  return LB_OK;
}


// Same contract as lb_flash_fwd (flash_attn.cu); head_dim 64 or 128, all pointers 16-byte
// aligned, token strides multiples of 8, causal needs Sk >= Sq.  Returns LB_ERR_SHAPE otherwise.
extern "C" int lb_flash_fwd_tc(const void* q, const void* k, const void* v, void* o, void* lse, int B, int Sq, int Sk,
                               int hq, int hkv, int d, long long q_ts, long long k_ts, long long v_ts, long long o_ts,
                               float scale, int causal, void* stream) {
  if (B <= 0 || Sq <= 0 || Sk <= 0 || hq % hkv) return LB_ERR_SHAPE;
  if ((q_ts | k_ts | v_ts | o_ts) % 8) return LB_ERR_SHAPE;
  if (causal && Sk < Sq) return LB_ERR_SHAPE;
  if (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)o) & 15) return LB_ERR_ARG;
  FaFwdParams p{(bf16*)o, (float*)lse, B, Sq, Sk, hq, hkv, o_ts, scale, causal, Sk, nullptr, 0u, 0};
  FaPush push;
  memset(&push, 0, sizeof(push));
  cudaStream_t s = (cudaStream_t)stream;
  switch (d) {
    case 64: return launch_fa_fwd<64>(q, k, v, p, push, q_ts, k_ts, v_ts, s);
    case 128: return launch_fa_fwd<128>(q, k, v, p, push, q_ts, k_ts, v_ts, s);
    default: return LB_ERR_SHAPE;
  }
}

// Warps per CTA of the forward kernel: every mover warp adds 1 to a key block's arrival word for K
// and 1 for V, so a block is complete at (calls so far) * 2 * this.
extern "C" int lb_flash_fwd_cp_mover_warps() { return FA_FWD_THREADS / 32; }

// Context-parallel forward: attention of q [B, Sq, hq, d] over the first Sk keys of the gather
// buffers kg / vg ([B, S_full, hkv*d] contiguous, this rank's peer-visible buffers), each 128-key
// block gated on `flags` [B][S_full/128] reaching `flag_target`.  With n_mov > 0 the same launch
// also pushes this rank's two zig-zag chunks of k_src / v_src ([B, 2*chunk_rows, hkv, d]) into
// every rank's buffers (kdst / vdst / flag_ptrs: host arrays of n_ranks pointers).
// chunk_rows must be a multiple of 128; S_full = 2 * n_ranks * chunk_rows.
extern "C" int lb_flash_fwd_cp(const void* q, const void* kg, const void* vg, void* o, void* lse, int B, int Sq, int Sk,
                               int S_full, int hq, int hkv, int d, long long q_ts, long long o_ts, float scale,
                               int causal, const void* flags, unsigned int flag_target, int n_mov, const void* k_src,
                               const void* v_src, long long k_ts, long long v_ts, int n_ranks, int rank,
                               void* const* kdst, void* const* vdst, void* const* flag_ptrs, int chunk_rows,
                               void* stream) {
  if (B <= 0 || Sq <= 0 || Sk <= 0 || Sk > S_full || hq % hkv || (S_full % 128)) return LB_ERR_SHAPE;
  if ((q_ts | o_ts) % 8) return LB_ERR_SHAPE;
  if (causal && Sk < Sq) return LB_ERR_SHAPE;
  FaFwdParams p{(bf16*)o, (float*)lse, B, Sq, Sk, hq, hkv, o_ts, scale, causal, S_full, (const unsigned int*)flags,
                flag_target, 0};
  FaPush push;
  memset(&push, 0, sizeof(push));
  if (n_mov > 0) {
    if (n_ranks < 1 || n_ranks > FA_MAX_RANKS || (chunk_rows % 128) || S_full != 2 * n_ranks * chunk_rows) return LB_ERR_SHAPE;
    if ((k_ts | v_ts) % 8) return LB_ERR_SHAPE;
    push.n_mov = n_mov; push.n_ranks = n_ranks; push.rank = rank; push.chunk_rows = chunk_rows; push.row_elems = hkv * d;
    push.k_src = (const bf16*)k_src; push.v_src = (const bf16*)v_src; push.k_ts = k_ts; push.v_ts = v_ts;
    for (int r = 0; r < n_ranks; r++) {
      push.k_dst[r] = (bf16*)kdst[r]; push.v_dst[r] = (bf16*)vdst[r]; push.flags[r] = (unsigned int*)flag_ptrs[r];
    }
  }
  cudaStream_t s = (cudaStream_t)stream;
  const long long kts = (long long)hkv * d;
  switch (d) {
    case 64: return launch_fa_fwd<64>(q, kg, vg, p, push, q_ts, kts, kts, s);
    case 128: return launch_fa_fwd<128>(q, kg, vg, p, push, q_ts, kts, kts, s);
    default: return LB_ERR_SHAPE;
  }
}
