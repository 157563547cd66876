// Grouped FP8 GEMM on tcgen05 for both expert GEMMs of the MoE shard.
//
// Replaces gemm_fp8_fp8_grouped_kernel / gemm_fp8_fp8_native_grouped_kernel
// (moe/solution/cuda/moe.cu:1373-1785, GEMM1) and gemm_fp32_fp8w_fused_acc_grouped_kernel
// (moe.cu:2186-2431, GEMM2); arithmetic contract from
// full-agent-pipeline/references/moe.py:95-118 (block scales) and :183-196 (the two matmuls).
//
// Orientation ("swap-AB"): the expert's weight rows are the 128-row M operand of
// the UMMA and the tokens are the N operand, so a batch of 1..128 tokens per
// expert streams every weight byte through shared memory exactly once per token
// tile and the tensor core does all fp8 decoding.  The operator is HBM-bound on
// the weight stream in every single-GPU regime, so the kernel is organised around
// keeping TMA loads of 16 KB weight tiles in flight:
//
//   warp 0  producer: TMA (SWIZZLE_128B, no multicast) of one weight tile
//           [128 rows x 128 K-bytes] and the token tile(s) [N_TILE x 128] per K-block
//           into a ring of STAGES shared-memory stages.
//   warps 1, 2  issuers (alternate stages): an elected lane issues the tcgen05.mma kind::f8f6f4 (M128, K32) of a
//           K-block into its own TMEM columns.  For GEMM2 the kNTerms e4m3 planes of
//           the token operand sit back to back in shared memory and, while they fit
//           N <= 256, are consumed as ONE operand of N = kNTerms * N_TILE rows, so the
//           weight tile is read from shared memory once per K32 step, not once per term.
//           G consecutive K-blocks form a hand-off group with one "full" barrier;
//           NBUF groups rotate through TMEM so that the hand-off latency between the
//           tensor core and the promotion warps is hidden.
//   warp 3  scales of every stage, copied asynchronously (cp.async) into a ring of slots behind the stage's own
//           "full" barrier, so that the promotion warps never wait for global memory.  Visible to them because the
//           issuer, which waited on "full", arrives on the stage's "done" barrier beside its commit.  A table of
//           scale products built by the promotion warps per item instead left 3000 to 7000 clocks per item without
//           a UMMA in flight, a third of GEMM2 at T = 512 (without it, and with the elected issue and the packed
//           arithmetic, calls are 1.07 times as fast at T = 512, 1.09 at T = 901, 1.08 at T = 64 on 16 experts).
//   warps 4-11 promotion + epilogue (two warps per TMEM lane quarter, each owning half
//           of the token columns): tcgen05.ld the partials of a group, release the TMEM
//           buffer, multiply by w_scale[e, m, kb] * b_scale[row, kb] and accumulate in
//           registers (the scales are arbitrary fp32 per 128-block, so they cannot ride
//           on the hardware's power-of-two block scaling); after the last K-block store
//           the fp32 tile transposed, i.e. token-major [row, m].  Packed two-element fp32 arithmetic
//           (add, mul, fma): T = 901 3 % faster than with scalar instructions.
//
// The token rows on the UMMA's M side (one scale per thread instead of one per column, GEMM2's planes stacked along
// M) is the faster arrangement in clocks and the slower one in time up to T = 1024: it multiplies M = 128 rows
// for tiles that have 5 to 40, and under the 1000 W cap the clock drops from 1.73 to 1.46 GHz (T = 512: 279 us).
//
// Work items (expert, weight-row tile, K-split, token tile) are decoded from the
// device-resident schedule; CTAs are persistent and take items round-robin.
// Every mbarrier wait is bounded (ptx.cuh); on a timeout the CTA records an error
// bit in the schedule block and leaves through the normal teardown.
#include "epilogue_device.cuh"
#include "gemm_common.cuh"

namespace moe {

namespace {

constexpr int kThreads = kGemmThreads;

template <int GEMM, int N_TILE>
struct Cfg {
  static constexpr int KB = GEMM == 1 ? kKB1 : kKB2;
  static constexpr int MT = GEMM == 1 ? kMT1 : kMT2;
  static constexpr int M_TOTAL = MT * 128;
  static constexpr int NTERMS = GEMM == 1 ? 1 : kNTerms;
  static constexpr bool STACK = NTERMS > 1 && NTERMS * N_TILE <= 256;   // planes consumed as one N operand
  static constexpr int N_MMA = STACK ? NTERMS * N_TILE : N_TILE;        // UMMA N
  static constexpr int MMA_PER_K4 = STACK ? 1 : NTERMS;
  static constexpr int PLANES = STACK ? NTERMS : 1;                     // column planes the epilogue sums
  static constexpr int KB_COLS = N_MMA;                                 // TMEM columns of one K-block partial
  // 128-token tiles run un-swapped: tokens are the UMMA M operand (TMEM lanes), weight rows the N operand
  // (TMEM columns).  A promotion thread then owns one token row, so the scale product of a K-block is ONE
  // value per thread instead of one per token column, and the result row is contiguous in memory.
  static constexpr bool TOK_ON_M = N_TILE == 128 && GEMM == 1;   // (GEMM2 measures the same either way)
  // Ragged token tiles (swapped orientation only): an item brings and multiplies the rows it has, rounded up to
  // RSTEP.  An SM takes in about 51 bytes per clock (large-batch GEMM1 at T = 4096 without its promotion: 48 KB K-blocks
  // in 962 clocks) and HBM delivers a 16 KB weight tile every ~700 clocks per SM, so a K-block may cost 35 KB of
  // operands before the weight stream stalls; with GEMM2's three planes a full 64-token tile makes it 40 KB.
  static constexpr int RSTEP = N_TILE >= 64 ? N_TILE / 4 : 16;
  static constexpr int RMAPS = N_TILE / RSTEP;
  static_assert(RMAPS >= 1 && RMAPS <= 4 && RSTEP % 16 == 0, "token maps per kernel / UMMA N granularity");
  static constexpr int A_BYTES = 128 * 128;
  static constexpr int B_BYTES = N_TILE * 128;
  static constexpr int KB_BYTES = A_BYTES + NTERMS * B_BYTES;           // operands of one K-block
  // K-blocks per pipeline stage.  A stage is also the TMEM hand-off unit: ONE tcgen05.commit per
  // stage tells the producer that the stage's shared memory is free and the promotion warps that
  // its partial sums are in TMEM.  (A commit costs the tensor pipe roughly 400 cycles, about as
  // much as six UMMAs of a 128-token tile, so two K-blocks share one wherever shared memory and
  // TMEM allow two stages of two.)
  static constexpr int KPS = (2 * KB_BYTES <= 64 * 1024 && 2 * KB_COLS <= 256) ? 2 : 1;
  static constexpr int G = KPS;
  static constexpr int CPW = N_TILE / 2;                                // token columns per epilogue warp
  static constexpr int STAGE_BYTES = KPS * KB_BYTES;
  // Scales of one stage: KPS x N_TILE row scales, then the KPS weight scales.
  static constexpr int SLOT_FLOATS = KPS * N_TILE + 4;
  static constexpr int AUX_BYTES = 1024;
  static constexpr int BUDGET = 227 * 1024 - 1024;   // 1 KB slack for the 1024-byte alignment of the ring
  static constexpr int STAGES_FIT = (BUDGET - 15 * SLOT_FLOATS * 4 - AUX_BYTES) / STAGE_BYTES;
  static constexpr int STAGES = STAGES_FIT > 10 ? 10 : STAGES_FIT;
  static constexpr int NBUF_FIT = 512 / (G * KB_COLS);
  // TMEM buffers (one stage of partials each).  Not more than shared-memory stages: the promotion warps
  // and the producer wait on the same per-stage barrier, and a stage must not complete a second phase
  // before the promotion warps have seen the first; the issuer is at most NBUF stages ahead of them.
  static constexpr int NBUF_CAP = NBUF_FIT > 4 ? 4 : NBUF_FIT;
  static constexpr int NBUF = NBUF_CAP > STAGES ? STAGES : NBUF_CAP;
  // A slot of scales is written again NSLOT stages later.  Its writer has then seen `done` of the stage STAGES before,
  // whose UMMAs waited for the promotion warps to release the buffer NBUF stages before that, after they had read
  // everything of the stages before that one.
  static constexpr int NSLOT = STAGES + NBUF + 1;
  static_assert(NSLOT <= 15, "scale slots counted in STAGES_FIT");
  static constexpr int SLOTS_BYTES = (NSLOT * SLOT_FLOATS * 4 + 127) / 128 * 128;
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + SLOTS_BYTES + AUX_BYTES + 1024;
  static constexpr int TMEM_USED = NBUF * G * KB_COLS;
  static constexpr int TMEM_COLS = TMEM_USED <= 32 ? 32 : TMEM_USED <= 64 ? 64 : TMEM_USED <= 128 ? 128
                                   : TMEM_USED <= 256 ? 256 : 512;
  static_assert(STAGES >= 2, "ring too small");
  static_assert(KB % KPS == 0 && (KPS & (KPS - 1)) == 0, "K-blocks per stage: a power of two dividing the K extent");
  static_assert(NBUF >= 2 && NBUF <= STAGES && TMEM_USED <= 512, "TMEM budget / ring depths");
  static_assert(N_MMA % 16 == 0 && N_MMA >= 16 && N_MMA <= 256, "invalid UMMA N for M = 128");
  static_assert(SMEM_BYTES > 116 * 1024, "one CTA per SM is assumed (TMEM is allocated without contention)");
};

struct Item {
  int e, m, s, row0, valid, kb0, kb1;
  int nv;      // token rows the item brings and multiplies: `valid` rounded up to the row step
};

template <int GEMM, int N_TILE>
__device__ __forceinline__ Item decode_item(int i, int split, const LaneSched& ls) {
  using C = Cfg<GEMM, N_TILE>;
  unsigned r, tiles_e;
  int off_e, cnt_e;
  Item it;
  ls.find(i, C::MT * split, it.e, r, tiles_e, off_e, cnt_e);
  int n = 0;
  it.s = 0;
  if (tiles_e > 1) {
    n = static_cast<int>(r % tiles_e);
    r /= tiles_e;
  }
  if (split > 1) {
    it.s = static_cast<int>(r % static_cast<unsigned>(split));
    r /= static_cast<unsigned>(split);
  }
  it.m = static_cast<int>(r);
  it.row0 = off_e + n * N_TILE;
  it.valid = min(N_TILE, cnt_e - n * N_TILE);
  it.nv = C::TOK_ON_M ? N_TILE : min(N_TILE, (it.valid + C::RSTEP - 1) / C::RSTEP * C::RSTEP);
  // split boundaries in units of one pipeline stage, so that no stage straddles two items
  constexpr int kUnits = C::KB / C::KPS;
  it.kb0 = ((it.s * kUnits) / split) * C::KPS;
  it.kb1 = (((it.s + 1) * kUnits) / split) * C::KPS;
  return it;
}

template <int GEMM, int N_TILE>
__global__ void __launch_bounds__(kThreads, 1)
grouped_gemm_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ TokenMaps tm_b, GemmArgs a) {
  using C = Cfg<GEMM, N_TILE>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  float* slots = reinterpret_cast<float*>(smem + C::STAGES * C::STAGE_BYTES);
  Aux* aux = reinterpret_cast<Aux*>(smem + C::STAGES * C::STAGE_BYTES + C::SLOTS_BYTES);

  const int warp = uniform_warp();
  const int lane = threadIdx.x & 31;
  griddep_launch_dependents();
  MoeSched* sched = a.sched;
  // everything that does not depend on earlier kernels first: barriers, descriptors, TMEM
  if (threadIdx.x == 0) {
    aux->abort = 0;
    for (int s = 0; s < C::STAGES; ++s) {
      mbar_init(smem_u32(&aux->full[s]), 1 + 32);     // the TMA producer and the 32 lanes of the scale warp
      mbar_init(smem_u32(&aux->done[s]), 2);          // the commit and the issuer's own arrival
    }
    for (int b = 0; b < C::NBUF; ++b) mbar_init(smem_u32(&aux->tempty[b]), kEpiWarps);
    fence_mbar_init();
    tma_prefetch_desc(&tm_w);
    for (int i = 0; i < C::RMAPS; ++i) tma_prefetch_desc(&tm_b.m[i]);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&aux->tmem_base), C::TMEM_COLS);
    tmem_relinquish();
  }
  griddep_wait();   // the schedule, the operands and the output slabs belong to earlier kernels until here
  const int items = __ldcg(GEMM == 1 ? &sched->items1 : &sched->items2);
  const int split = __ldcg(GEMM == 1 ? &sched->split1 : &sched->split2);
  const int n_sel_pad = __ldcg(&sched->n_sel_pad);
  LaneSched ls;
  ls.load(GEMM == 1 ? sched->tile_prefix : sched->tile_prefix2, sched->offs, lane);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = aux->tmem_base;
  volatile int* abort_flag = &aux->abort;
  const uint32_t smem_base = smem_u32(smem);
  const uint32_t full_base = smem_u32(&aux->full[0]), done_base = smem_u32(&aux->done[0]);
  const uint32_t tempty_base = smem_u32(&aux->tempty[0]);
  uint32_t stage = 0, ph = 0, buf = 0, bph = 0;      // ring positions, advanced the same way by every role
  auto advance = [&]() {
    if (++stage == C::STAGES) { stage = 0; ph ^= 1u; }
    if (++buf == C::NBUF) { buf = 0; bph ^= 1u; }
  };

  if (warp < kFirstEpiWarp) {
    bool ok = true;
    if (warp == 0) {
      // ---------------------------------------------------------------- TMA producer (an elected lane issues)
      for (int i = blockIdx.x; ok && i < items; i += gridDim.x) {
        const Item w = decode_item<GEMM, N_TILE>(i, split, ls);
        const int wy = w.e * C::M_TOTAL + w.m * 128;
        const uint32_t tx = C::KPS * (C::A_BYTES + C::NTERMS * w.nv * 128);
        const CUtensorMap* mb = &tm_b.m[w.nv / C::RSTEP - 1];
        for (int kb = w.kb0; kb < w.kb1; kb += C::KPS) {
          if (!mbar_wait(done_base + stage * 8, ph ^ 1u, abort_flag)) { ok = false; break; }
          if (elect_one()) {
            const uint32_t bar = full_base + stage * 8;
            mbar_arrive_expect_tx(bar, tx);
            const uint32_t dst = smem_base + stage * C::STAGE_BYTES;
            // weights: [KPS][128 rows][128 B]; tokens: [KPS][NTERMS planes][nv rows][128 B]
            tma_load_3d(dst, &tm_w, 0, wy, kb, bar);
            if (GEMM == 1) tma_load_3d(dst + C::KPS * C::A_BYTES, mb, 0, w.row0, kb, bar);
            else tma_load_4d(dst + C::KPS * C::A_BYTES, mb, 0, w.row0, 0, kb, bar);
          }
          advance();
        }
      }
    } else if (warp == 3) {
      // ---------------------------------------------------------------- scales of every stage
      // The promotion warps only multiply; nothing between two items makes them wait for global memory.
      uint32_t slot = smem_u32(slots);
      const uint32_t slot_end = slot + C::NSLOT * C::SLOT_FLOATS * 4;
      for (int i = blockIdx.x; ok && i < items; i += gridDim.x) {
        const Item w = decode_item<GEMM, N_TILE>(i, split, ls);
        const float* wsp = a.w_scale + (static_cast<size_t>(w.e) * C::MT + w.m) * C::KB;
        for (int kb = w.kb0; kb < w.kb1; kb += C::KPS) {
          if (!mbar_wait(done_base + stage * 8, ph ^ 1u, abort_flag)) { ok = false; break; }
#pragma unroll
          for (int g = 0; g < C::KPS; ++g) {
            const float* bsp = a.b_scale + static_cast<size_t>(kb + g) * a.rows_cap;
#pragma unroll
            for (int j0 = 0; j0 < N_TILE; j0 += 32)    // rows past the tile's last one: any value, their columns are dropped
              if (j0 < w.nv)
                cp_async4(slot + (g * N_TILE + j0 + lane) * 4, bsp + min(w.row0 + j0 + lane, a.rows_cap - 1));
          }
          if (lane < C::KPS) cp_async4(slot + (C::KPS * N_TILE + lane) * 4, wsp + kb + lane);
          cp_async_arrive(full_base + stage * 8);
          slot += C::SLOT_FLOATS * 4;
          if (slot == slot_end) slot = smem_u32(slots);
          advance();
        }
      }
    } else {
      // ---------------------------------------------------------------- UMMA issuers (warps 1 and 2, an elected lane issues)
      // They take alternate stages.  A stage's UMMAs only touch that stage's shared memory and TMEM columns and each issuer
      // commits its own, so stages are independent; with one issuer the waits and loop overhead between two stages
      // (~500 cycles) leave the tensor pipe idle, because the queue behind it is only an instruction or two deep.
      const uint64_t desc_const = umma_desc_k_sw128(0);          // everything but the start address
      int nst = 0;
      for (int i = blockIdx.x; ok && i < items; i += gridDim.x) {
        const Item w = decode_item<GEMM, N_TILE>(i, split, ls);
        const uint32_t idesc = umma_idesc_e4m3(128, C::STACK ? C::NTERMS * w.nv : w.nv);
        const uint32_t plane_bytes = static_cast<uint32_t>(w.nv) * 128;
        for (int kb = w.kb0; kb < w.kb1; kb += C::KPS, ++nst, advance()) {   // items span whole stages
          if ((nst & 1) != warp - 1) continue;             // the other issuer's stage
          if (!mbar_wait(tempty_base + buf * 8, bph ^ 1u, abort_flag)) { ok = false; break; }
          if (!mbar_wait(full_base + stage * 8, ph, abort_flag)) { ok = false; break; }
          tc_fence_after_sync();
          if (elect_one()) {
            const uint32_t sbase = smem_base + stage * C::STAGE_BYTES;
#pragma unroll
            for (int u = 0; u < C::KPS; ++u) {
              const uint64_t adesc = desc_const | ((sbase + u * C::A_BYTES) >> 4);
              const uint32_t sb = sbase + C::KPS * C::A_BYTES + u * (C::NTERMS * plane_bytes);
              const uint32_t d = tmem_base + buf * (C::G * C::KB_COLS) + u * C::KB_COLS;
#pragma unroll
              for (int t = 0; t < C::MMA_PER_K4; ++t) {
                const uint64_t bdesc = desc_const | ((sb + t * plane_bytes) >> 4);
#pragma unroll
                for (int k4 = 0; k4 < 4; ++k4) {  // +32 bytes of K inside the 128-byte swizzle atom = +2 encoded units
                  if constexpr (C::TOK_ON_M) umma_f8(d, bdesc + 2 * k4, adesc + 2 * k4, idesc, (t | k4) != 0 ? 1u : 0u);
                  else umma_f8(d, adesc + 2 * k4, bdesc + 2 * k4, idesc, (t | k4) != 0 ? 1u : 0u);
                }
              }
            }
            umma_commit(done_base + stage * 8);
            // The promotion warps read the stage's scales behind `done` and never wait on `full`.  The commit orders the
            // UMMAs; this arrival releases what the issuer acquired with `full`, the copied scales among it.
            mbar_arrive(done_base + stage * 8);
          }
        }
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ promotion + epilogue (warps 4..11)
    const int q = warp & 3;                       // TMEM lane quarter this warp may access
    const int h = (warp - kFirstEpiWarp) >> 2;    // which half of the token columns
    const uint32_t lane_addr = static_cast<uint32_t>(q * 32) << 16;
    int slot = 0;
    bool ok = true;
    auto release = [&]() {
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(tempty_base + buf * 8);
    };
    for (int i = blockIdx.x; ok && i < items; i += gridDim.x) {
      const Item w = decode_item<GEMM, N_TILE>(i, split, ls);
      float acc[C::CPW];
#pragma unroll
      for (int j = 0; j < C::CPW; ++j) acc[j] = 0.0f;

      for (int kb = w.kb0; kb < w.kb1; kb += C::KPS, advance()) {
        if (!mbar_wait(done_base + stage * 8, ph, abort_flag)) { ok = false; break; }
        tc_fence_after_sync();
        const uint32_t taddr = tmem_base + lane_addr + buf * (C::G * C::KB_COLS) + h * C::CPW;
        const float* sl = slots + slot * C::SLOT_FLOATS;
        if (++slot == C::NSLOT) slot = 0;
        if constexpr (C::TOK_ON_M) {
          static_assert(C::PLANES == 1 && C::CPW == 64 && C::KB_COLS == 128, "un-swapped path: one 128 x 128 partial per K-block");
          // lane = token row (row0 + 32 q + lane), columns = this warp's half of the 128 weight rows
#pragma unroll
          for (int g = 0; g < C::G; ++g) {
            float v[C::CPW];
            tmem_ld32(taddr + g * C::KB_COLS, v);
            tmem_ld32(taddr + g * C::KB_COLS + 32, v + 32);
            const float f = sl[C::KPS * N_TILE + g] * sl[g * N_TILE + q * 32 + lane];
            tmem_wait_ld();
            if (g == C::G - 1) release();
            fma_scaled<C::CPW>(acc, v, f);
          }
        } else {
          // Every partial of the stage is read back before the buffer is released and the arithmetic starts.  The
          // stacked planes are w.nv columns apart.  A warp whose columns start past the item's rows reads nothing (they
          // are never stored).
          static_assert(C::G * C::PLANES * C::CPW <= 96, "the partials of a stage must fit the registers");
          const bool live = h * C::CPW < w.nv;
          float v[C::G][C::PLANES][C::CPW];
          if (live) {
#pragma unroll
            for (int g = 0; g < C::G; ++g)
#pragma unroll
              for (int p = 0; p < C::PLANES; ++p) tmem_ld_cols<C::CPW>(taddr + g * C::KB_COLS + p * w.nv, v[g][p]);
            tmem_wait_ld();
          }
          release();
          if (!live) continue;
#pragma unroll
          for (int g = 0; g < C::G; ++g) {
            const float ws = sl[C::KPS * N_TILE + g];
            const float4* scv = reinterpret_cast<const float4*>(sl + g * N_TILE + h * C::CPW);
#pragma unroll
            for (int u = 0; u < C::CPW / 4; ++u) {
              const float4 f = scv[u];
              const float2 f2[2] = {__fmul2_rn(make_float2(f.x, f.y), make_float2(ws, ws)),
                                    __fmul2_rn(make_float2(f.z, f.w), make_float2(ws, ws))};
#pragma unroll
              for (int x = 0; x < 2; ++x) {
                const int c = u * 4 + 2 * x;
                float2 sum = make_float2(v[g][C::PLANES - 1][c], v[g][C::PLANES - 1][c + 1]);
#pragma unroll
                for (int p = C::PLANES - 2; p >= 0; --p) sum = __fadd2_rn(sum, make_float2(v[g][p][c], v[g][p][c + 1]));   // smallest terms first
                const float2 r = __ffma2_rn(sum, f2[x], make_float2(acc[c], acc[c + 1]));
                acc[c] = r.x;
                acc[c + 1] = r.y;
              }
            }
          }
        }
      }
      if (!ok) break;
      if constexpr (C::TOK_ON_M) {
        if (q * 32 + lane < w.valid) {      // one token row, 64 consecutive outputs
          float* out = a.out + (static_cast<size_t>(w.s) * n_sel_pad + w.row0 + q * 32 + lane) * C::M_TOTAL + w.m * 128 + h * C::CPW;
#pragma unroll
          for (int j = 0; j < C::CPW / 8; ++j) st_global_v8(out + 8 * j, acc + 8 * j);   // whole 32-byte sectors
        }
      } else {
        float* out = a.out + (static_cast<size_t>(w.s) * n_sel_pad + w.row0 + h * C::CPW) * C::M_TOTAL + w.m * 128 +
                     q * 32 + lane;
#pragma unroll
        for (int j = 0; j < C::CPW; ++j)
          if (h * C::CPW + j < w.valid) out[static_cast<size_t>(j) * C::M_TOTAL] = acc[j];
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

template <int GEMM, int N_TILE>
int launch_one(const CUtensorMap& tm_w, const TokenMaps& tm_b, const GemmArgs& a, int ctas, cudaStream_t stream) {
  using C = Cfg<GEMM, N_TILE>;
  return static_cast<int>(launch_pdl(grouped_gemm_kernel<GEMM, N_TILE>, dim3(ctas), dim3(kThreads), C::SMEM_BYTES,
                                     stream, tm_w, tm_b, a));
}

template <int GEMM, int N_TILE>
int init_one() {
  using C = Cfg<GEMM, N_TILE>;
  return static_cast<int>(cudaFuncSetAttribute(grouped_gemm_kernel<GEMM, N_TILE>,
                                               cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES));
}

}  // namespace


int grouped_gemm_kblocks_per_stage(int gemm_id, int n_tile) {
#define MOE_CASE(G, N) \
  if (gemm_id == G && n_tile == N) return Cfg<G, N>::KPS;
  MOE_CASE(1, 32) MOE_CASE(1, 64) MOE_CASE(1, 128)
  MOE_CASE(2, 32) MOE_CASE(2, 64) MOE_CASE(2, 128)
#undef MOE_CASE
  return 1;
}

int grouped_gemm_init() {
  int rc = 0;
  if ((rc = init_one<1, 32>())) return rc;
  if ((rc = init_one<1, 64>())) return rc;
  if ((rc = init_one<1, 128>())) return rc;
  if ((rc = init_one<2, 32>())) return rc;
  if ((rc = init_one<2, 64>())) return rc;
  if ((rc = init_one<2, 128>())) return rc;
  return 0;
}

int grouped_gemm_row_step(int n_tile) { return n_tile >= 64 ? n_tile / 4 : 16; }

int launch_grouped_gemm(int gemm_id, int n_tile, const CUtensorMap& tm_w, const TokenMaps& tm_b, const GemmArgs& a,
                        int ctas, cudaStream_t stream) {
#define MOE_CASE(G, N) \
  if (gemm_id == G && n_tile == N) return launch_one<G, N>(tm_w, tm_b, a, ctas, stream);
  MOE_CASE(1, 32) MOE_CASE(1, 64) MOE_CASE(1, 128)
  MOE_CASE(2, 32) MOE_CASE(2, 64) MOE_CASE(2, 128)
#undef MOE_CASE
  return static_cast<int>(cudaErrorInvalidValue);
}

}  // namespace moe
