// Large-batch grouped FP8 GEMMs (more than 1024 tokens per call: 128-token tiles) with the
// stages around them fused into the epilogues.
//
//   GEMM1 + SwiGLU:  replaces gemm_fp8_fp8_grouped_kernel + swiglu_kernel of the reference
//     (moe/solution/cuda/moe.cu:1373-1785, 2125-2167).  The fp32 GEMM1 result never exists in memory:
//     one work item owns a (128-token tile, 128-column block jb of the SwiGLU output) pair; its weight
//     operand is 256 rows made of TWO 128-row TMA boxes, rows [jb*128, +128) of the first half of W13
//     and the same rows of the second half, so that x1 and x2 of the same 128 output columns meet in
//     one 128 x 256 accumulator tile (UMMA N = 256).  After the K loop a thread holds
//     C = silu(x2) * x1 (full-agent-pipeline/references/moe.py:187-193: the SECOND half goes through
//     silu) of its token row, the four threads of a row agree on the block's power-of-two scale, and C
//     goes out as the three e4m3 planes + scale that GEMM2 reads.  The wide tile is also what the
//     hardware wants: an SM takes in about 51 bytes per clock (48 KB K-blocks in 962 clocks at T = 4096,
//     without the promotion), a 128 x 128 x 128 fp8 tile needs
//     32 KB per 256 tensor-pipe clocks (128 B / clock), a 128 x 256 tile 48 KB per 512 (96 B / clock).
//   GEMM2 (+ combine):  replaces gemm_fp32_fp8w_fused_acc_grouped_kernel and fin_cast8_kernel
//     (moe.cu:2186-2431, 2473-2496).  COMBINE = false stores fp32 rows for the deterministic
//     combine kernel (ascending expert order, the order of references/moe.py:196-200).
//     COMBINE = true is the reference's own scheme (moe.cu:2404-2430): the epilogue multiplies by
//     the routing weight and adds into an fp32 [T, 7168] accumulator with 16-byte vector
//     reductions; a counter per (token, 128-column tile) tells the LAST contributor, which casts
//     the finished 128 columns to bf16 and writes them to the output.  No thread ever waits for
//     another one, but the fp32 summation order is whatever the hardware makes it.
//
// Orientation: the token tile is the UMMA M operand (TMEM lanes), the weight rows the N operand
// (TMEM columns), so a promotion thread owns ONE token row and the 128-block scale product of a
// K-block is one value per thread: f = a_scale[row, kb] * w_scale[e, block, kb].  The scales are
// arbitrary fp32, so every K-block is accumulated into its own TMEM columns and promoted with one
// FMA per element (they cannot ride on the hardware's power-of-two block scaling).
//
// Roles (640 threads, one CTA per SM):
//   warp 0      TMA producer (one elected lane; SWIZZLE_128B boxes, no multicast).  Weights and token planes have rings
//               of their own: a K-block of GEMM2 is 80 KB, two whole ones are all that fits, and then the load of one
//               is exposed behind the UMMAs of the other; one plane at a time, 2.3 to 3 K-blocks are in flight.  A
//               ragged token tile brings the rows it has (boxes of 1 to 4 times 32 rows); the rows behind them are
//               whatever the slot held before, and their lanes of the accumulator are never read.
//   warps 1, 2  UMMA issuers (one elected lane each, alternate K-blocks)
//   warp 3      scales of every K-block, copied asynchronously into a ring in shared memory behind the K-block's own
//               barrier: the promotion warps' loads from global memory were a round trip in every K-block
//   warps 4-19  promotion + epilogue: four warps per TMEM lane quarter, each owning a quarter of the
//               accumulator columns.  Sixteen warps (four per scheduler) so that the TMEM read-back
//               latency of one warp is covered by the FMAs of the others; with eight the read-back
//               latency was exposed in every K-block and the tensor pipe sat idle two thirds of the time.
// The two rings, the scale warp, the ragged boxes and the elected lanes together: T = 4096 778 -> 695 us per call,
// T = 14107 1644 -> 1475 us, the 256-expert layer at T = 16384 15.3 -> 13.9 ms (per call, both builds in turn; the
// kernels alone at T = 4096: GEMM1 341 -> 279 us, GEMM2 288 -> 252).
// Every wait is bounded (ptx.cuh); a timeout raises the CTA's abort flag, all roles fall through to
// the normal teardown (TMEM freed) and an error bit is left in the schedule block.
#include "epilogue_device.cuh"
#include "kernels.h"
#include "ptx.cuh"

namespace moe {
namespace {

constexpr int kRowStep = kLargeRowStep;
constexpr int kLEpiWarps = 16;
constexpr int kLFirstEpi = 4;
constexpr int kLEpiThreads = kLEpiWarps * 32;
constexpr int kLThreads = (kLFirstEpi + kLEpiWarps) * 32;   // 640
// setmaxnreg: the launch allocates kLRegsAtLaunch per thread (65536 / 640 rounded down to 8); the control
// warpgroup gives registers away, the four promotion warpgroups take them.
constexpr int kLRegsAtLaunch = 96;
constexpr int kLRegsControl = 32;
constexpr int kLRegsEpi = 112;
static_assert(128 * kLRegsControl + kLEpiThreads * kLRegsEpi <= kLRegsAtLaunch * kLThreads,
              "register reallocation would never complete");

template <int GEMM>
struct LCfg {
  static constexpr int KB = GEMM == 1 ? kKB1 : kKB2;             // K-blocks of the contraction
  static constexpr int J = GEMM == 1 ? kKB2 : kMT2 / 2;          // weight-side units per token tile: 16 / 28
  static constexpr int NTERMS = GEMM == 1 ? 1 : kNTerms;         // e4m3 planes of the token operand
  static constexpr int W_ROWS = 256;                             // weight rows of an item = UMMA N = TMEM columns per K-block
  static constexpr int W_BYTES = W_ROWS * 128;                   // one K-block of the weight operand
  static constexpr int TOK_BYTES = 128 * 128;                    // one K-block of 128 token rows (one plane)
  // Two rings: one K-block of weights per slot, one PLANE of a K-block of tokens per slot.  A slot is free as soon as
  // the four UMMAs of its plane (weights: of the K-block's last plane) have completed.
  static constexpr int WS = GEMM == 1 ? 4 : 3;
  static constexpr int PS = GEMM == 1 ? 4 : 7;
  static constexpr int BUF_COLS = W_ROWS;                        // TMEM columns of one K-block's partial sums
  static constexpr int NBUF = 2;
  static constexpr int TMEM_COLS = 512;
  // Scales of one K-block: 128 row scales, then the two weight scales of the item's 256 weight rows.  A slot is written
  // again NSLOT K-blocks later; its writer has then seen K-block WS before complete, whose UMMAs waited for the
  // promotion warps to release the buffer of NBUF before that, after they had read that K-block's scales.
  static constexpr int SLOT_FLOATS = 128 + 4;
  static constexpr int NSLOT = WS + NBUF + 1;
  static constexpr int SLOTS_BYTES = (NSLOT * SLOT_FLOATS * 4 + 127) / 128 * 128;
  static constexpr int AUX_BYTES = 4096;
  static constexpr int RING_BYTES = WS * W_BYTES + PS * TOK_BYTES;
  static constexpr int SMEM_BYTES = RING_BYTES + SLOTS_BYTES + AUX_BYTES + 1024;
  static_assert(NBUF * BUF_COLS <= TMEM_COLS, "TMEM ring");
  // A `pdone` phase must be seen by everybody before its slot's next one completes: the promotion warps are at most
  // NBUF K-blocks behind the issuers, and the plane that completes the next phase is PS planes later.
  static_assert(PS >= NBUF * NTERMS && PS >= NTERMS && WS >= NBUF, "ring depths");
  // The producer waits for K-block n - WS before it loads K-block n's weights, on the barrier of that K-block's last
  // plane: the next plane on that barrier must not be loaded before, i.e. not belong to an earlier K-block than n.
  static_assert(NTERMS - 1 + PS >= WS * NTERMS, "a weight slot's barrier must still show the phase that is waited for");
  static_assert(SMEM_BYTES <= 227 * 1024 && SMEM_BYTES > 116 * 1024, "one CTA per SM");
};

struct LAux {
  uint64_t wfull[4];       // TMA and the scale warp -> issuers: a K-block's weights (GEMM1: and tokens) and scales
  uint64_t pfull[8];       // TMA -> issuers: one plane of tokens (GEMM2)
  uint64_t pdone[8];       // issuers -> producer, scale warp, promotion warps: the UMMAs of a plane have completed
  uint64_t tempty[2];      // promotion warps -> issuers
  uint64_t esync;          // all promotion threads meet (bounded replacement of a named barrier)
  uint32_t tmem_base;
  int abort;
  int prefix[kELocal + 1];
  int offs[kELocal + 1];
  float amax[4][128];      // per column group and token row: |C| maximum of the thread's columns
};
static_assert(sizeof(LAux) <= 4096, "LAux must fit its slot");

// A position in a ring of N slots and the parity of its round.
template <int N>
struct Pos {
  uint32_t i = 0, ph = 0;
  __device__ __forceinline__ void step(uint32_t k = 1) {
    i += k;
    if (i >= N) { i -= N; ph ^= 1u; }
  }
};

struct LItem {
  int e, j, row0, valid;
};

// Item i -> (expert, weight-side unit j, token tile); token tiles of one weight unit are adjacent, so that
// CTAs working at the same time read the same weight rows (they come from HBM once, then from L2).
template <int GEMM>
__device__ __forceinline__ LItem decode_large(int i, const LAux* aux) {
  constexpr int J = LCfg<GEMM>::J;
  int e = 0;   // largest e with prefix[e] * J <= i (experts without tiles repeat the prefix value)
#pragma unroll 1
  for (int k = 16; k > 0; k >>= 1)
    if (e + k < kELocal && aux->prefix[e + k] * J <= i) e += k;
  const int r = i - aux->prefix[e] * J;
  const int tiles_e = aux->prefix[e + 1] - aux->prefix[e];
  const int n = r % tiles_e;
  LItem it;
  it.e = e;
  it.j = r / tiles_e;
  const int cnt = aux->offs[e + 1] - aux->offs[e];
  it.row0 = aux->offs[e] + n * 128;
  it.valid = min(128, cnt - n * 128);
  return it;
}

__device__ __forceinline__ void red_add_v4(float* p, float x, float y, float z, float w) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(x), "f"(y), "f"(z), "f"(w) : "memory");
}

template <int GEMM, bool COMBINE>
__global__ void __launch_bounds__(kLThreads, 1)
grouped_gemm_large_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ TokenMaps tm_b,
                          const __grid_constant__ GemmArgs a) {
  using C = LCfg<GEMM>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  float* slots = reinterpret_cast<float*>(smem + C::RING_BYTES);
  LAux* aux = reinterpret_cast<LAux*>(smem + C::RING_BYTES + C::SLOTS_BYTES);

  const int warp = uniform_warp();
  const int lane = threadIdx.x & 31;
  griddep_launch_dependents();
  MoeSched* sched = a.sched;
  // everything that does not depend on earlier kernels first: barriers, descriptors, TMEM
  if (threadIdx.x == 0) {
    aux->abort = 0;
    for (int s = 0; s < C::WS; ++s) mbar_init(smem_u32(&aux->wfull[s]), 1 + 32);   // the producer and the scale warp's lanes
    for (int s = 0; s < C::PS; ++s) {
      mbar_init(smem_u32(&aux->pfull[s]), 1);
      mbar_init(smem_u32(&aux->pdone[s]), 2);      // the commit and the issuer's own arrival
    }
    for (int b = 0; b < C::NBUF; ++b) mbar_init(smem_u32(&aux->tempty[b]), kLEpiWarps);
    mbar_init(smem_u32(&aux->esync), kLEpiThreads);
    fence_mbar_init();
    tma_prefetch_desc(&tm_w);
    for (int i = 0; i < 4; ++i) tma_prefetch_desc(&tm_b.m[i]);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&aux->tmem_base), C::TMEM_COLS);
    tmem_relinquish();
  }
  griddep_wait();   // the schedule, the operands and the outputs belong to earlier kernels until here
  const int items = GEMM == 1 ? sched->items1 : sched->items2;
  if (threadIdx.x <= kELocal) {
    aux->prefix[threadIdx.x] = GEMM == 1 ? sched->tile_prefix[threadIdx.x] : sched->tile_prefix2[threadIdx.x];
    aux->offs[threadIdx.x] = sched->offs[threadIdx.x];
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = aux->tmem_base;
  volatile int* abort_flag = &aux->abort;
  const uint32_t smem_base = smem_u32(smem), tok_base = smem_base + C::WS * C::W_BYTES;
  const uint32_t wfull_base = smem_u32(&aux->wfull[0]), pfull_base = smem_u32(&aux->pfull[0]);
  const uint32_t pdone_base = smem_u32(&aux->pdone[0]), tempty_base = smem_u32(&aux->tempty[0]);
  constexpr bool JOINT = C::NTERMS == 1;      // tokens and weights of a K-block on one barrier

  if (warp < kLFirstEpi) {
    setmaxnreg_dec<kLRegsControl>();
    bool ok = true;
    Pos<C::WS> wp;
    Pos<C::PS> pp, old;        // next plane; last plane of the K-block that used the weight slot before
    old.step(C::NTERMS - 1);
    if (warp == 0) {
      // ------------------------------------------------------------------ TMA producer
      int n = 0;
      for (int i = blockIdx.x; ok && i < items; i += gridDim.x) {
        const LItem w = decode_large<GEMM>(i, aux);
        const int steps = (w.valid + kRowStep - 1) / kRowStep;      // a ragged tile brings the rows it has
        const CUtensorMap* mb = &tm_b.m[steps - 1];
        const uint32_t tok_tx = static_cast<uint32_t>(steps) * (kRowStep * 128);
#pragma unroll 1
        for (int kb = 0; kb < C::KB; ++kb, ++n, wp.step()) {
          if (n >= C::WS) {
            if (!mbar_wait_hot(pdone_base + old.i * 8, old.ph, abort_flag)) { ok = false; break; }
            old.step(C::NTERMS);
          }
          if (elect_one()) {
            const uint32_t bar = wfull_base + wp.i * 8;
            const uint32_t dst = smem_base + wp.i * C::W_BYTES;
            mbar_arrive_expect_tx(bar, C::W_BYTES + (JOINT ? tok_tx : 0u));
            if constexpr (GEMM == 1) {
              // weights: 128 rows of the first half of W13 | the same 128 rows of the second half
              const int y = w.e * k2I + w.j * 128;
              tma_load_3d(dst, &tm_w, 0, y, kb, bar);
              tma_load_3d(dst + 128 * 128, &tm_w, 0, y + kI, kb, bar);
              tma_load_3d(tok_base + pp.i * C::TOK_BYTES, mb, 0, w.row0, kb, bar);
            } else {
              tma_load_3d(dst, &tm_w, 0, w.e * kH + w.j * 256, kb, bar);                  // 256 weight rows as two boxes
              tma_load_3d(dst + 128 * 128, &tm_w, 0, w.e * kH + w.j * 256 + 128, kb, bar);
            }
          }
          if constexpr (JOINT) {
            pp.step();
          } else {
            for (int t = 0; t < C::NTERMS; ++t, pp.step()) {
              if (!mbar_wait_hot(pdone_base + pp.i * 8, pp.ph ^ 1u, abort_flag)) { ok = false; break; }
              if (elect_one()) {
                const uint32_t bar = pfull_base + pp.i * 8;
                mbar_arrive_expect_tx(bar, tok_tx);
                tma_load_4d(tok_base + pp.i * C::TOK_BYTES, mb, 0, w.row0, t, kb, bar);
              }
            }
            if (!ok) break;
          }
        }
      }
    } else if (warp == 3) {
      // ------------------------------------------------------------------ scales of every K-block
      uint32_t slot = smem_u32(slots);
      const uint32_t slot_end = slot + C::NSLOT * C::SLOT_FLOATS * 4;
      int n = 0;
      for (int i = blockIdx.x; ok && i < items; i += gridDim.x) {
        const LItem w = decode_large<GEMM>(i, aux);
        // the two 128-row weight blocks of the item: GEMM1 j and j + 16, GEMM2 2 j and 2 j + 1
        const float* wsp = a.w_scale + (GEMM == 1 ? (static_cast<size_t>(w.e) * kMT1 + w.j + (lane & 1) * kKB2) * kKB1
                                                  : (static_cast<size_t>(w.e) * kMT2 + 2 * w.j + (lane & 1)) * kKB2);
#pragma unroll 1
        for (int kb = 0; kb < C::KB; ++kb, ++n, wp.step()) {
          if (n >= C::WS) {
            if (!mbar_wait_hot(pdone_base + old.i * 8, old.ph, abort_flag)) { ok = false; break; }
            old.step(C::NTERMS);
          }
          const float* bsp = a.b_scale + static_cast<size_t>(kb) * a.rows_cap;
#pragma unroll
          for (int j0 = 0; j0 < 128; j0 += 32)    // rows past the tile's last one: any value, they are dropped
            if (j0 < w.valid) cp_async4(slot + (j0 + lane) * 4, bsp + min(w.row0 + j0 + lane, a.rows_cap - 1));
          if (lane < 2) cp_async4(slot + (128 + lane) * 4, wsp + kb);
          cp_async_arrive(wfull_base + wp.i * 8);
          slot += C::SLOT_FLOATS * 4;
          if (slot == slot_end) slot = smem_u32(slots);
        }
      }
    } else {
      // ------------------------------------------------------------------ UMMA issuers (alternate K-blocks)
      constexpr uint32_t idesc = umma_idesc_e4m3(128, C::W_ROWS);
      const uint64_t desc_const = umma_desc_k_sw128(0);
      Pos<C::NBUF> tb;
      int n = 0;
      for (int i = blockIdx.x; ok && i < items; i += gridDim.x) {
#pragma unroll 1
        for (int s = 0; s < C::KB; ++s, ++n) {
          if ((n & 1) == warp - 1) {
            if (!mbar_wait_hot(tempty_base + tb.i * 8, tb.ph ^ 1u, abort_flag)) { ok = false; break; }
            if (!mbar_wait_hot(wfull_base + wp.i * 8, wp.ph, abort_flag)) { ok = false; break; }
            const uint64_t wdesc = desc_const | ((smem_base + wp.i * C::W_BYTES) >> 4);
            const uint32_t d = tmem_base + tb.i * C::BUF_COLS;
#pragma unroll
            for (int t = 0; t < C::NTERMS; ++t, pp.step()) {
              if constexpr (!JOINT) {
                if (!mbar_wait_hot(pfull_base + pp.i * 8, pp.ph, abort_flag)) { ok = false; break; }
              }
              tc_fence_after_sync();
              if (elect_one()) {
                const uint64_t tdesc = desc_const | ((tok_base + pp.i * C::TOK_BYTES) >> 4);
#pragma unroll
                for (int k4 = 0; k4 < 4; ++k4)   // +32 bytes of K inside the 128-byte swizzle atom = +2 encoded units
                  umma_f8(d, tdesc + 2 * k4, wdesc + 2 * k4, idesc, (t | k4) != 0 ? 1u : 0u);
                umma_commit(pdone_base + pp.i * 8);
                // the promotion warps read the K-block's scales behind `pdone` alone: this arrival releases to them what
                // the issuer acquired with `wfull` (see grouped_gemm.cu)
                mbar_arrive(pdone_base + pp.i * 8);
              }
            }
            if (!ok) break;
          } else {
            pp.step(C::NTERMS);
          }
          wp.step();
          tb.step();
        }
      }
    }
    __syncwarp();   // block-wide barriers below need whole warps
  } else {
    setmaxnreg_inc<kLRegsEpi>();
    // ------------------------------------------------------------------ promotion + epilogue (warps 4..19)
    const int q = warp & 3;                       // TMEM lane quarter this warp may access
    const int cg = (warp - kLFirstEpi) >> 2;      // column group: a quarter of the accumulator columns
    const int trow = q * 32 + lane;               // token row inside the tile
    const uint32_t lane_addr = static_cast<uint32_t>(q * 32) << 16;
    Pos<C::PS> last;                              // last plane of the next K-block
    last.step(C::NTERMS - 1);
    Pos<C::NBUF> tb;
    int slot = 0;
    auto release = [&]() {
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(tempty_base + tb.i * 8);
    };
    uint32_t eph = 0;
    bool ok = true;
    auto epi_sync = [&]() {
      mbar_arrive(smem_u32(&aux->esync));
      if (!mbar_wait_hot(smem_u32(&aux->esync), eph, abort_flag)) ok = false;
      eph ^= 1u;
    };
    for (int i = blockIdx.x; ok && i < items; i += gridDim.x) {
      const LItem w = decode_large<GEMM>(i, aux);
      const int row = w.row0 + trow;
      float acc[64];      // GEMM1: [0, 32) x1 of this thread's 32 columns, [32, 64) x2 of the same; GEMM2: 64 columns
#pragma unroll
      for (int x = 0; x < 64; ++x) acc[x] = 0.0f;
      const bool live = q * 32 < w.valid;         // a warp whose rows lie past the tile's last one reads nothing
#pragma unroll 1
      for (int s = 0; s < C::KB; ++s, last.step(C::NTERMS), tb.step()) {
        if (!mbar_wait_hot(pdone_base + last.i * 8, last.ph, abort_flag)) { ok = false; break; }
        tc_fence_after_sync();
        const float* sl = slots + slot * C::SLOT_FLOATS;
        if (++slot == C::NSLOT) slot = 0;
        if (!live) { release(); continue; }
        const uint32_t taddr = tmem_base + lane_addr + tb.i * C::BUF_COLS + cg * (GEMM == 1 ? 32 : 64);
        float v[32];
        tmem_ld32(taddr, v);
        // GEMM1: the halves belong to two weight blocks; GEMM2: this thread's 64 columns lie in one, 2 j + (cg >> 1)
        const float nb = sl[trow];
        const float f1 = sl[128 + (GEMM == 1 ? 0 : cg >> 1)] * nb;
        const float f2 = GEMM == 1 ? sl[129] * nb : f1;
        tmem_wait_ld();
        fma_scaled<32>(acc, v, f1);
        tmem_ld32(taddr + (GEMM == 1 ? 128 : 32), v);
        tmem_wait_ld();
        release();
        fma_scaled<32>(acc + 32, v, f2);
      }
      if (!ok) break;
      if constexpr (GEMM == 1) {
        float amax = 0.0f;
#pragma unroll
        for (int x = 0; x < 32; ++x) {
          acc[x] = swiglu_value(acc[x], acc[32 + x]);
          amax = fmaxf(amax, fabsf(acc[x]));
        }
        aux->amax[cg][trow] = amax;
        epi_sync();      // the four threads of a row have published their maxima
        if (!ok) break;
        amax = fmaxf(fmaxf(aux->amax[0][trow], aux->amax[1][trow]), fmaxf(aux->amax[2][trow], aux->amax[3][trow]));
        const int ex = plane_scale_exponent(amax);
        const float inv = __uint_as_float(static_cast<uint32_t>(127 - ex) << 23);
        if (trow < w.valid) {
          uint32_t pk[kNTerms][8];
#pragma unroll
          for (int x = 0; x < 32; ++x) {
            uint8_t t3[kNTerms];
            split_e4m3_terms(acc[x] * inv, t3);
#pragma unroll
            for (int t = 0; t < kNTerms; ++t) {
              if ((x & 3) == 0) pk[t][x >> 2] = 0;
              pk[t][x >> 2] |= static_cast<uint32_t>(t3[t]) << (8 * (x & 3));
            }
          }
#pragma unroll
          for (int t = 0; t < kNTerms; ++t) {
            uint4* dst = reinterpret_cast<uint4*>(a.cq + (static_cast<size_t>(t) * a.rows_cap + row) * kI + w.j * kBlock + cg * 32);
            dst[0] = make_uint4(pk[t][0], pk[t][1], pk[t][2], pk[t][3]);
            dst[1] = make_uint4(pk[t][4], pk[t][5], pk[t][6], pk[t][7]);
          }
          if (cg == 0) a.c_scale[static_cast<size_t>(w.j) * a.rows_cap + row] = __uint_as_float(static_cast<uint32_t>(ex + 127) << 23);
        }
      } else {
        const int tile = 2 * w.j + (cg >> 1);     // the 128-row weight block of this thread's columns
        if (trow < w.valid) {
          const int col0 = w.j * 256 + cg * 64;
          if constexpr (!COMBINE) {
            float* out = a.out + static_cast<size_t>(row) * kH + col0;
#pragma unroll
            for (int x = 0; x < 8; ++x) st_global_v8(out + 8 * x, acc + 8 * x);   // whole 32-byte sectors
          } else {
            const int t = __ldcg(a.perm_token + row);
            const float pw = __ldcg(a.perm_weight + row);
            float* dst = a.acc32 + static_cast<size_t>(t) * kH + col0;
#pragma unroll
            for (int x = 0; x < 16; ++x)
              red_add_v4(dst + 4 * x, __fmul_rn(acc[4 * x], pw), __fmul_rn(acc[4 * x + 1], pw), __fmul_rn(acc[4 * x + 2], pw),
                         __fmul_rn(acc[4 * x + 3], pw));
            __threadfence();      // the reductions above are performed before the arrival below is
            const int target = 2 * __popc(__ldcg(a.local_mask + t));   // two threads per (row, 128-column tile)
            const int old = atomicAdd(a.tile_cnt + static_cast<size_t>(t) * kMT2 + tile, 1);
            if (old == target - 1) {
              // last contributor of (token, column tile): all 128 sums are complete
              __threadfence();
              const float4* src = reinterpret_cast<const float4*>(a.acc32 + static_cast<size_t>(t) * kH + tile * 128);
              uint16_t* orow = (a.out_rows ? a.out_rows[t] : a.out_bf16 + static_cast<size_t>(t) * kH) + tile * 128;
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                float4 u[16];
#pragma unroll
                for (int x = 0; x < 16; ++x) u[x] = __ldcg(src + h * 16 + x);
#pragma unroll
                for (int x = 0; x < 8; ++x) {
                  uint4 o;
                  o.x = pack_bf16x2(u[2 * x].x, u[2 * x].y);
                  o.y = pack_bf16x2(u[2 * x].z, u[2 * x].w);
                  o.z = pack_bf16x2(u[2 * x + 1].x, u[2 * x + 1].y);
                  o.w = pack_bf16x2(u[2 * x + 1].z, u[2 * x + 1].w);
                  reinterpret_cast<uint4*>(orow)[h * 8 + x] = o;
                }
              }
            }
          }
        }
      }
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (threadIdx.x == 0 && aux->abort) atomicOr(&sched->status, GEMM == 1 ? kErrGemm1Timeout : kErrGemm2Timeout);
  if (warp == 1) {
    if (aux->abort) settle_after_abort();
    __syncwarp();
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, C::TMEM_COLS);
  }
}

// Before a GEMM2 launch with the fused combine: clears the fp32 accumulator and the arrival counters, and
// writes the output rows of tokens without a local expert (all zeros; nobody else will).
__global__ void __launch_bounds__(256) combine_prepare_kernel(float4* acc, size_t n_vec, const uint32_t* local_mask, int T,
                                                              uint16_t* out_bf16, uint16_t* const* out_rows) {
  griddep_launch_dependents();
  griddep_wait();
  const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n_vec;
       i += static_cast<size_t>(gridDim.x) * blockDim.x)
    acc[i] = z;
  for (int t = blockIdx.x; t < T; t += gridDim.x) {
    if (local_mask[t] != 0) continue;
    uint4* row = reinterpret_cast<uint4*>(out_rows ? out_rows[t] : out_bf16 + static_cast<size_t>(t) * kH);
    for (int c = threadIdx.x; c < kH * 2 / 16; c += blockDim.x) row[c] = make_uint4(0u, 0u, 0u, 0u);
  }
}

template <int GEMM, bool COMBINE>
int init_large() {
  return static_cast<int>(cudaFuncSetAttribute(grouped_gemm_large_kernel<GEMM, COMBINE>,
                                               cudaFuncAttributeMaxDynamicSharedMemorySize, LCfg<GEMM>::SMEM_BYTES));
}

}  // namespace

int grouped_gemm_large_init() {
  int rc = 0;
  if ((rc = init_large<1, false>())) return rc;
  if ((rc = init_large<2, false>())) return rc;
  if ((rc = init_large<2, true>())) return rc;
  return 0;
}

int launch_grouped_gemm_large(int gemm_id, bool fused_combine, const CUtensorMap& tm_w, const TokenMaps& tm_b,
                              const GemmArgs& a, int ctas, cudaStream_t stream) {
  if (gemm_id == 1)
    return static_cast<int>(launch_pdl(grouped_gemm_large_kernel<1, false>, dim3(ctas), dim3(kLThreads),
                                       LCfg<1>::SMEM_BYTES, stream, tm_w, tm_b, a));
  if (fused_combine)
    return static_cast<int>(launch_pdl(grouped_gemm_large_kernel<2, true>, dim3(ctas), dim3(kLThreads),
                                       LCfg<2>::SMEM_BYTES, stream, tm_w, tm_b, a));
  return static_cast<int>(launch_pdl(grouped_gemm_large_kernel<2, false>, dim3(ctas), dim3(kLThreads), LCfg<2>::SMEM_BYTES,
                                     stream, tm_w, tm_b, a));
}

int launch_combine_prepare(float* acc32, size_t acc_floats, const uint32_t* local_mask, int T, uint16_t* out_bf16,
                           uint16_t* const* out_rows, cudaStream_t stream) {
  const size_t n_vec = acc_floats / 4;
  size_t blocks = (n_vec + 255) / 256;
  if (blocks > 16 * kNumSMs) blocks = 16 * kNumSMs;
  if (blocks < 1) blocks = 1;
  return static_cast<int>(launch_pdl(combine_prepare_kernel, dim3(static_cast<unsigned>(blocks)), dim3(256), 0, stream,
                                     reinterpret_cast<float4*>(acc32), n_vec, local_mask, T, out_bf16, out_rows));
}

}  // namespace moe
