// Grouped-expert GEMMs of the quantised encodings for many routes per expert: D[weight row, route] = W_e . x^T, wide tiles.
//
// Same contract, operands and order of sums as grouped.cu and grouped_ts.cu (the bits are theirs).  What bounds a 256 x 256
// tile whose converted weights lie in shared memory is shared-memory bandwidth: per 64 k the tensor core reads 96 KB of
// operands, the conversion writes 32 KB and the copies 40 KB, 176 KB against 128 bytes a clock.  Here the converted weights are
// the A operand in TENSOR MEMORY, as in grouped_ts.cu, under a tile as wide as tensor memory allows beside it:
//
//  * 256 weight rows (two M = 128 halves) x up to 192 routes: 384 columns of float32 sums and two stages of 64 k of converted
//    weights.  Per 64 k the tensor core reads the activation tile twice (48 KB), the copies write it once (24 KB) and the codes
//    cost 16 KB: 88 KB in 768 tensor clocks.
//  * Eight conversion warps (a thread owns a weight row, codes -> BF16 -> tcgen05.st) and sixteen epilogue warps of their own, so that the conversion of the next tile starts under the epilogue; four warps copying activation rows by index
//    (gate/up) or one lane issuing TMA boxes (down); a weight TMA lane; the MMA issuer.  One CTA per SM.
//  * A gate and its up row sit in the same lane of the two halves: SwiGLU needs no exchange.  Results are transposed
//    through shared memory, 16 (8) routes at a time, and leave as one bulk copy of 256 (512) contiguous bytes per route.
//  * The weight ring of the down GEMM starts to fill while the gate/up GEMM's last CTAs still run.
//
// Measured (B200, OLMoE Q4, 1024 tokens = 128 routes per expert, whole operator): 197 us on 256-row tiles, 159 here; where the
// lines lie stands at grouped_gemm_takes_wide.  With eight epilogue warps instead of sixteen 168 (8192 tokens: 975 | 897), with
// 128-route tiles and four stages of weights 205.  What bounds it: a step of 64 k takes about 900 clocks even with 16 routes,
// in the hand-overs between copying, converting and multiplying warps, and the accumulators are drained between tiles.
#include "grouped.cuh"

#include <cuda.h>

#include "common.cuh"
#include "tc.cuh"

namespace umaq {
namespace {

constexpr int kRows = 128;                // weight rows of a half = lanes of an MMA
constexpr int NW = kTileCapWide;          // routes of a tile
constexpr int kStepK = 64;                // one 128-byte swizzle atom of BF16
constexpr int kActBox = 16;               // rows of an activation TMA box
constexpr int kWideMaxGroups = 16;        // K <= 2048
constexpr int kCopyWarps = 4, kConvertWarps = 8, kEpilogueWarps = 16;
constexpr int kCopyThreads = kCopyWarps * 32;
constexpr int kFirstCopy = 2, kFirstConvert = kFirstCopy + kCopyWarps, kFirstEpilogue = kFirstConvert + kConvertWarps;
constexpr int kWideThreads = (kFirstEpilogue + kEpilogueWarps) * 32;
constexpr int kGroups = kEpilogueWarps / 4, kGroupThreads = 128;      // epilogue groups of four warps
constexpr int kBTile = NW * kStepK * 2, kBStages = 4;
constexpr int kAStages = 2, kAHalfCols = kStepK / 2, kAStageCols = 2 * kAHalfCols, kACol = 2 * NW;
constexpr int kWideTmemCols = 512;
static_assert(kACol + kAStages * kAStageCols <= kWideTmemCols, "tensor memory");
constexpr int kScaleBuffer = 2 * kRows * kWideMaxGroups;               // floats
constexpr int kStageBuffer = 4096;        // an epilogue chunk: 16 routes x 128 columns or 8 x 256 of BF16

template <int ENC>
struct WideShape {
  static constexpr int kPackedRow = ENC == ENC_Q4 ? kStepK / 2 : kStepK;   // code bytes of a row and step
  static constexpr int kHalfBytes = kRows * kPackedRow, kWeightBytes = 2 * kHalfBytes;
  static constexpr int kPStages = ENC == ENC_Q4 ? 6 : 4;
};

template <int ENC>
struct WideShared {
  using S = WideShape<ENC>;
  uint64_t in_full[kBStages], in_empty[kBStages];
  uint64_t p_full[S::kPStages], p_empty[S::kPStages];
  uint64_t a_full[kAStages], a_empty[kAStages];
  uint64_t sc_full[2], sc_empty[2];
  uint64_t acc_full, acc_empty;
  uint32_t tmem_base;
  int abort_flag;
  int row[NW];
};
template <int ENC>
constexpr size_t wide_smem_bytes() {
  return (size_t)kBStages * kBTile + (size_t)WideShape<ENC>::kPStages * WideShape<ENC>::kWeightBytes + 2 * kScaleBuffer * 4 +
         2 * kGroups * kStageBuffer + sizeof(WideShared<ENC>);
}

struct WideTile {
  int col, expert, row0, nrows;
};
// The table is read through L2: the down GEMM's weight warp looks at it before its programmatic wait.
__device__ __forceinline__ WideTile wide_tile(const GroupedParams& p, int it, int n_col) {
  WideTile t;
  const int m = it / n_col;
  t.col = it - m * n_col;
  t.expert = __ldcg(p.tile_expert + m); t.row0 = __ldcg(p.tile_row0 + m); t.nrows = __ldcg(p.tile_rows + m);
  return t;
}
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[16]) { tmem_ld16(taddr, r); }
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[8]) { tmem_ld8(taddr, r); }
// `bytes` contiguous bytes shared -> global on this thread's bulk async-group
__device__ __forceinline__ void bulk_s2g(void* dst, const void* src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(smem_u32(src)), "r"(bytes) : "memory");
}

template <int ENC, int MODE>
__global__ void __launch_bounds__(kWideThreads, 1)
grouped_wide_kernel(const __grid_constant__ CUtensorMap map_act, const __grid_constant__ CUtensorMap map_w0,
                    const __grid_constant__ CUtensorMap map_w1, const GroupedParams p) {
  using S = WideShape<ENC>;
  constexpr int kPStages = S::kPStages;
  constexpr int kFeatures = MODE == 0 ? kRows : 2 * kRows;                // output columns of a tile
  constexpr int kChunk = kStageBuffer / (2 * kFeatures);                  // routes of an epilogue chunk
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* sB = smem_raw;                                                 // [activation stages]
  uint8_t* sP = sB + kBStages * kBTile;                                   // [code stages]
  uint8_t* sOut = sP + kPStages * S::kWeightBytes;                        // [groups][2][routes][columns]
  float* sScales = reinterpret_cast<float*>(sOut + 2 * kGroups * kStageBuffer);     // [2][256 rows][groups]
  WideShared<ENC>& sh = *reinterpret_cast<WideShared<ENC>*>(sScales + 2 * kScaleBuffer);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int K = p.k;
  const int nk = K / kStepK, groups = K >> 7;
  const int n_col = p.n_rows / kFeatures;
  const int first = blockIdx.x, step = gridDim.x;
  volatile int* abort_flag = &sh.abort_flag;

  if (tid == 0) {
    for (int s = 0; s < kBStages; ++s) { mbar_init(&sh.in_full[s], MODE == 0 ? kCopyThreads : 1); mbar_init(&sh.in_empty[s], 1); }
    for (int s = 0; s < kPStages; ++s) { mbar_init(&sh.p_full[s], 1); mbar_init(&sh.p_empty[s], kConvertWarps); }
    for (int s = 0; s < kAStages; ++s) { mbar_init(&sh.a_full[s], kConvertWarps); mbar_init(&sh.a_empty[s], 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(&sh.sc_full[s], 1); mbar_init(&sh.sc_empty[s], kConvertWarps); }
    mbar_init(&sh.acc_full, 1);
    mbar_init(&sh.acc_empty, kEpilogueWarps);
    sh.abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 0) {
    tmem_alloc(&sh.tmem_base, kWideTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sh.tmem_base;
  // The gate/up kernel lets the down kernel start only after its own wait: whoever runs in the down kernel then finds the
  // tile table complete, and the weight warp (which reads nothing else that a kernel wrote) need not wait there.
  if (MODE == 0 || warp != 1) pdl_wait();
  pdl_launch_dependents();
  const int total = __ldcg(p.num_tiles) * n_col;
  auto fail = [&]() { atomicExch(p.status, (unsigned)ERR_DEVICE_TIMEOUT); *abort_flag = 1; };

  if (warp == 0) {
    // ===================== MMA issuer: the warp stays converged, one elected lane issues ==========
    Ring<kBStages> rb;
    Ring<kAStages> ra;
    uint32_t seq = 0;
    const uint64_t b_desc0 = smem_desc_sw128(smem_u32(sB));
    for (int it = first; it < total; it += step, ++seq) {
      if (warp_sees(abort_flag)) break;
      const WideTile t = wide_tile(p, it, n_col);
      const int n16 = (t.nrows + 15) & ~15;
      // kind::f16, BF16 x BF16 -> FP32, K-major operands, M = 128, N = the tile's routes
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n16 >> 3) << 17) | (8u << 24);
      bool ok = seq == 0 || mbar_wait_warp(&sh.acc_empty, (seq - 1) & 1);
      for (int kc = 0; kc < nk; ++kc) {
        ok = __all_sync(0xffffffffu, ok && mbar_wait(&sh.in_full[rb.slot], rb.phase) && mbar_wait(&sh.a_full[ra.slot], ra.phase));
        if (!ok) break;
        tc_fence_after();
        if (MODE == 0) fence_proxy_async();
        if (elect_one()) {
          const uint64_t bd = b_desc0 + (uint64_t)(rb.slot * (kBTile >> 4));          // descriptors count 16-byte units
          const uint32_t a_tmem = tmem + kACol + ra.slot * kAStageCols;
#pragma unroll
          for (int half = 0; half < 2; ++half)
#pragma unroll
            for (int k = 0; k < kStepK / 16; ++k)
              tc_mma_bf16_ts(tmem + half * NW, a_tmem + half * kAHalfCols + k * 8, bd + k * 2, idesc, k ? 1u : (uint32_t)(kc != 0));
          tc_commit(&sh.a_empty[ra.slot]);
          tc_commit(&sh.in_empty[rb.slot]);
          if (kc == nk - 1) tc_commit(&sh.acc_full);
        }
        __syncwarp();
        rb.next();
        ra.next();
      }
      if (!ok) { if (lane == 0) fail(); break; }
    }
  } else if (warp == 1) {
    // ===================== TMA producer: scales and packed weight rows ===========================
    // The whole warp waits (a lone lane's wait takes twice as long and slows the others'), one lane issues.
    {
      uint32_t kidx = 0, seq = 0;
      Ring<kPStages> rp;
      for (int it = first; it < total; it += step) {
        if (warp_sees(abort_flag)) break;
        const WideTile t = wide_tile(p, it, n_col);
        const long long wrow0 = (long long)t.expert * p.n_rows + t.col * kFeatures;
        const uint32_t sb = seq & 1;
        if (!__all_sync(0xffffffffu, seq < 2 || mbar_wait(&sh.sc_empty[sb], ((seq >> 1) - 1) & 1))) { if (lane == 0) fail(); break; }
        if (lane == 0) {
          float* dst_sc = sScales + sb * kScaleBuffer;
          const uint32_t bytes = (uint32_t)kRows * groups * 4;
          mbar_expect_tx(&sh.sc_full[sb], 2 * bytes);
          bulk_g2s(dst_sc, p.scales0 + wrow0 * groups, bytes, &sh.sc_full[sb]);
          bulk_g2s(dst_sc + kRows * groups, MODE == 0 ? p.scales1 + wrow0 * groups : p.scales0 + (wrow0 + kRows) * groups, bytes,
                   &sh.sc_full[sb]);
        }
        __syncwarp();
        ++seq;
        bool ok = true;
        for (int kc = 0; kc < nk; ++kc, ++kidx, rp.next()) {
          const uint32_t s = rp.slot;
          ok = __all_sync(0xffffffffu, kidx < (uint32_t)kPStages || mbar_wait(&sh.p_empty[s], rp.phase ^ 1));
          if (!ok) break;
          if (lane == 0) {
            mbar_expect_tx(&sh.p_full[s], S::kWeightBytes);
            uint8_t* dst = sP + s * S::kWeightBytes;
            tma_load_2d(dst, &map_w0, kc * S::kPackedRow, (int)wrow0, &sh.p_full[s]);
            if (MODE == 0) tma_load_2d(dst + S::kHalfBytes, &map_w1, kc * S::kPackedRow, (int)wrow0, &sh.p_full[s]);
            else tma_load_2d(dst + S::kHalfBytes, &map_w0, kc * S::kPackedRow, (int)wrow0 + kRows, &sh.p_full[s]);
          }
          __syncwarp();
        }
        if (!ok) { if (lane == 0) fail(); break; }
      }
      if (*abort_flag) {                                // nobody consumes: wait (bounded) for the copies in flight
        for (uint32_t q = seq > 2 ? seq - 2 : 0; q < seq; ++q) mbar_wait(&sh.sc_full[q & 1], (q >> 1) & 1);
        for (uint32_t k2 = kidx > (uint32_t)kPStages ? kidx - kPStages : 0; k2 < kidx; ++k2)
          mbar_wait(&sh.p_full[k2 % kPStages], (k2 / kPStages) & 1);
      }
    }
  } else if (warp < kFirstConvert) {
    if (MODE == 1) {
      // ===================== TMA producer: activation rows in sorted order =========================
      if (warp == kFirstCopy) {
        uint32_t kidx = 0;
        Ring<kBStages> rb;
        for (int it = first; it < total; it += step) {
          if (warp_sees(abort_flag)) break;
          const WideTile t = wide_tile(p, it, n_col);
          const int boxes = (t.nrows + kActBox - 1) / kActBox;
          bool ok = true;
          for (int kc = 0; kc < nk; ++kc, ++kidx, rb.next()) {
            const uint32_t s = rb.slot;
            ok = __all_sync(0xffffffffu, kidx < (uint32_t)kBStages || mbar_wait(&sh.in_empty[s], rb.phase ^ 1));
            if (!ok) break;
            if (lane == 0) mbar_expect_tx(&sh.in_full[s], boxes * kActBox * 128);
            __syncwarp();
            if (lane < boxes)
              tma_load_2d(sB + s * kBTile + lane * kActBox * 128, &map_act, kc * kStepK, t.row0 + lane * kActBox, &sh.in_full[s]);
            __syncwarp();
          }
          if (!ok) { if (lane == 0) fail(); break; }
        }
        if (*abort_flag)
          for (uint32_t k2 = kidx > (uint32_t)kBStages ? kidx - kBStages : 0; k2 < kidx; ++k2)
            mbar_wait(&sh.in_full[k2 % kBStages], (k2 / kBStages) & 1);
      }
    } else {
      // ===================== activation rows by index: 128 threads write every tile =================
      // As in grouped.cu: thread j copies 16-byte chunk j & 7 of rows (j >> 3) + 16 i into the 128-byte-swizzled slot, so
      // eight neighbouring lanes read one row's 128 contiguous bytes.  Rows up to the next multiple of 16 are zero-filled.
      const int pt = tid - kFirstCopy * 32;                 // 0 .. 127
      const int c = pt & 7, rbase = pt >> 3;                // rows rbase + 16 i: all have r & 7 == rbase & 7
      const uint32_t dst_off = (uint32_t)rbase * 128 + (uint32_t)((c ^ (rbase & 7)) << 4);
      uint32_t kidx = 0;
      Ring<kBStages> rb;
      bool ok = true;
      for (int it = first; it < total; it += step) {
        // everybody has read the previous tile's rows, and the threads agree whether to go on
        if (named_bar_or(1, kCopyThreads, !ok || *abort_flag != 0)) break;
        const WideTile t = wide_tile(p, it, n_col);
        const int n16 = (t.nrows + 15) >> 4;                // runs of 16 rows
        for (int r = pt; r < NW; r += kCopyThreads) sh.row[r] = r < t.nrows ? p.gather_route[t.row0 + r] / p.gather_top_k : -1;
        named_bar_sync(1, kCopyThreads);
        int tok[NW / 16];
#pragma unroll
        for (int i = 0; i < NW / 16; ++i) tok[i] = sh.row[rbase + 16 * i];
        const uint8_t* col = reinterpret_cast<const uint8_t*>(p.gather_src) + c * 16;
        for (int kc = 0; kc < nk; ++kc, ++kidx, rb.next(), col += kStepK * 2) {
          ok = __all_sync(0xffffffffu, kidx < (uint32_t)kBStages || mbar_wait(&sh.in_empty[rb.slot], rb.phase ^ 1));
          if (!ok) break;
          uint8_t* dst = sB + rb.slot * kBTile + dst_off;
#pragma unroll
          for (int i = 0; i < NW / 16; ++i)
            if (i < n16) cp_async16(dst + i * 2048, col + (size_t)(tok[i] < 0 ? 0 : tok[i]) * K * 2, tok[i] >= 0);
          cp_async_arrive(&sh.in_full[rb.slot]);            // when they have landed; the issuer fences them towards the tensor core
        }
      }
      if (!ok && lane == 0) fail();
      cp_async_commit();
      cp_async_wait<0>();                                   // also on the abort path: nothing of this thread stays in flight
    }
  } else if (warp < kFirstEpilogue) {
    // ===================== conversion warps: packed codes -> BF16 rows of A in tensor memory =========
    // A thread owns one row = one lane of one half.
    const int quarter = warp & 3, half = (warp - kFirstConvert) >> 2;
    const int row = half * kRows + quarter * 32 + lane;
    const uint32_t a_lane = tmem + ((uint32_t)(quarter * 32) << 16) + kACol + half * kAHalfCols;
    const bool vec = (groups & 3) == 0;
    uint32_t kidx = 0, seq = 0;
    Ring<kPStages> rp;
    Ring<kAStages> ra;
    for (int it = first; it < total; it += step) {
      const uint32_t sbuf = seq & 1;
      mbar_wait_or_flag(&sh.sc_full[sbuf], (seq >> 1) & 1, abort_flag);
      ++seq;
      const float* sc = sScales + sbuf * kScaleBuffer + row * groups;
      float4 s4 = make_float4(0.f, 0.f, 0.f, 0.f);
      Q4Scale qs = q4_scale(0.f);
      for (int kc = 0; kc < nk; ++kc, ++kidx) {
        if (vec) {                                          // rows 64 bytes apart: four scales per load, a quarter of the conflicts
          if ((kc & 7) == 0) s4 = *reinterpret_cast<const float4*>(sc + (kc >> 1));
        } else if ((kc & 1) == 0) {
          s4.x = s4.y = s4.z = s4.w = sc[kc >> 1];
        }
        const int j4 = (kc >> 1) & 3;
        const float scale = j4 < 2 ? (j4 == 0 ? s4.x : s4.y) : (j4 == 2 ? s4.z : s4.w);
        mbar_wait_or_flag(&sh.p_full[rp.slot], rp.phase, abort_flag);
        const uint8_t* src = sP + rp.slot * S::kWeightBytes + row * S::kPackedRow;
        if (ENC == ENC_Q4 && (kc & 1) == 0) qs = q4_scale(scale);
        const bool fused = ENC == ENC_Q4 && __all_sync(0xffffffffu, qs.fused);
#pragma unroll
        for (int j = 0; j < 2; ++j) {                       // 32 k each, the first under the wait for the stage
          uint32_t out[16];
          if (ENC == ENC_Q4) {
            const uint4 raw = *reinterpret_cast<const uint4*>(src + j * 16);
            if (fused) convert_q4_fused(raw, qs, out);
            else convert_q4(raw, scale, out);
          } else {                                          // 64-byte rows, TMA swizzle: 16-byte chunk ^ (row >> 1 & 3)
            const int sw = (row >> 1) & 3;
            convert_q8(*reinterpret_cast<const uint4*>(src + (((2 * j) ^ sw) << 4)),
                       *reinterpret_cast<const uint4*>(src + (((2 * j + 1) ^ sw) << 4)), scale, out);
          }
          if (j == 0) {
            if (kidx >= (uint32_t)kAStages) mbar_wait_or_flag(&sh.a_empty[ra.slot], ra.phase ^ 1, abort_flag);
            tc_fence_after();
          }
          tmem_st16(a_lane + ra.slot * kAStageCols + j * 16, out);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh.p_empty[rp.slot]);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh.a_full[ra.slot]);
        rp.next();
        ra.next();
      }
      if (warp_sees(abort_flag)) { if (lane == 0) fail(); break; }
      if (lane == 0) mbar_arrive(&sh.sc_empty[sbuf]);
    }
  } else {
    // ===================== epilogue warps ========================================================
    // Lane = weight row of either half, column = route; the groups of four warps take the chunks of routes in turn.  A
    // chunk is written to shared memory route by route (a warp's 32 lanes 64 contiguous bytes) and leaves as one bulk copy
    // per route; a group has two buffers, and its first warp waits for the reads of the one filled last before the group's
    // barrier, so that after the barrier the other one is free to be filled.
    const int quarter = warp & 3, group = (warp - kFirstEpilogue) >> 2;
    const int row = quarter * 32 + lane;
    const uint32_t lane_base = tmem + ((uint32_t)(quarter * 32) << 16);
    // word order of a run of 8 features that a quantised down GEMM expects: (f0,f4)(f1,f5)(f2,f6)(f3,f7)
    const int at = MODE == 0 && p.permute_out ? (row & ~7) + 2 * (row & 3) + ((row >> 2) & 1) : row;
    uint8_t* const buffers = sOut + group * 2 * kStageBuffer;
    uint32_t seq = 0, filled = 0;
    bool ok = true;
    for (int it = first; it < total; it += step, ++seq) {
      const WideTile t = wide_tile(p, it, n_col);
      ok = mbar_wait_warp(&sh.acc_full, seq & 1);
      // the group's warps agree whether to go on: none may be left waiting at a chunk's barrier
      if (named_bar_or(2 + group, kGroupThreads, !ok || *abort_flag != 0)) break;
      tc_fence_after();
      const int chunks = (t.nrows + kChunk - 1) / kChunk;
      for (int c = group; c < chunks; c += kGroups, ++filled) {
        const int left = min(kChunk, t.nrows - c * kChunk);
        const long long r0 = (long long)t.row0 + c * kChunk;
        __nv_bfloat16* stage = reinterpret_cast<__nv_bfloat16*>(buffers + (filled & 1) * kStageBuffer);
        uint32_t a[kChunk], b[kChunk];
        tmem_ld(lane_base + c * kChunk, a);
        tmem_ld(lane_base + NW + c * kChunk, b);
        tmem_ld_wait();
        if (c + kGroups >= chunks) {                              // this warp's last reads of the tile
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&sh.acc_empty);
        }
        if (MODE == 0) {
#pragma unroll
          for (int j = 0; j < kChunk; ++j)
            stage[j * kRows + at] = __float2bfloat16_rn(silu_f32(__uint_as_float(a[j])) * __uint_as_float(b[j]));
        } else {
          const float wr = lane < left ? p.route_weight[r0 + lane] : 0.f;
#pragma unroll
          for (int j = 0; j < kChunk; ++j) {
            const float w = __shfl_sync(0xffffffffu, wr, j);
            stage[j * 2 * kRows + row] = __float2bfloat16_rn(__uint_as_float(a[j]) * w);
            stage[j * 2 * kRows + kRows + row] = __float2bfloat16_rn(__uint_as_float(b[j]) * w);
          }
        }
        fence_proxy_async();                                // this thread's staging writes -> visible to the copy engine
        if (quarter == 0) bulk_wait_read<0>();              // (the first warp's lanes issue the copies)
        named_bar_sync(2 + group, kGroupThreads);
        if (quarter == 0) {
          if (lane < left) bulk_s2g(p.out + (r0 + lane) * p.out_stride + t.col * kFeatures, stage + lane * kFeatures, kFeatures * 2);
          bulk_commit();
        }
      }
      if (group >= chunks && lane == 0) mbar_arrive(&sh.acc_empty);      // fewer chunks than groups
    }
    if (!ok && lane == 0) fail();
    if (quarter == 0) bulk_wait_all();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem, kWideTmemCols);
  }
}

template <int ENC, int MODE>
int launch_wide(const GroupedGemmArgs& a, const GroupedParams& p, cudaStream_t stream) {
  using S = WideShape<ENC>;
  auto kernel = grouped_wide_kernel<ENC, MODE>;
  constexpr size_t smem = wide_smem_bytes<ENC>();
  static_assert(smem <= 227 * 1024, "shared memory of an SM");
  static thread_local int configured = -1;
  int dev = 0;
  cudaGetDevice(&dev);
  if (configured != dev) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) { set_error("grouped: cudaFuncSetAttribute: %s", cudaGetErrorString(e)); return ERR_LAUNCH; }
    configured = dev;
  }
  CUtensorMap ma, m0, m1;
  const uint64_t wrows = (uint64_t)a.num_experts * a.n_rows, rowb = ENC == ENC_Q4 ? a.k / 2 : a.k;
  const CUtensorMapSwizzle swz = ENC == ENC_Q4 ? CU_TENSOR_MAP_SWIZZLE_NONE : CU_TENSOR_MAP_SWIZZLE_64B;
  if (!make_map(&m0, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, a.w0, rowb, wrows, S::kPackedRow, kRows, swz) ||
      !make_map(&m1, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, MODE == 0 ? a.w1 : a.w0, rowb, wrows, S::kPackedRow, kRows, swz))
    return ERR_LAUNCH;
  // with rows fetched by index `act` is [tokens, k] and the map is never used: any valid map will do
  if (!make_map(&ma, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, a.act, (uint64_t)a.k, (uint64_t)(MODE == 0 ? kActBox : a.total_rows),
                kStepK, kActBox, CU_TENSOR_MAP_SWIZZLE_128B))
    return ERR_LAUNCH;
  const cudaError_t e = launch_chained(kernel, dim3(sm_count()), dim3(kWideThreads), smem, stream, ma, m0, m1, p);
  if (e != cudaSuccess) { set_error("grouped: launch failed: %s", cudaGetErrorString(e)); return ERR_LAUNCH; }
  return ERR_NONE;
}

}  // namespace

// Both GEMMs of a layer, the down GEMM directly behind the gate/up GEMM on the stream (its weight warp relies on it).
int launch_grouped_gemm_wide(const GroupedGemmArgs& a, cudaStream_t stream) {
  if (a.k % 128 || a.k > kWideMaxGroups * 128 || a.n_rows % (a.mode == 0 ? kRows : 2 * kRows) || a.total_rows <= 0 ||
      a.max_tiles <= 0 || a.tile_cap > NW || (a.mode == 0 ? !a.gather_route || a.gather_top_k < 1 : !a.route_weight)) {
    set_error("grouped: unsupported shape (k %d, rows per expert %d)", a.k, a.n_rows);
    return ERR_BAD_ARGUMENT;
  }
  GroupedParams p{};
  p.k = a.k; p.n_rows = a.n_rows;
  p.scales0 = a.s0; p.scales1 = a.s1;
  p.num_tiles = a.num_tiles; p.tile_expert = a.tile_expert; p.tile_row0 = a.tile_row0; p.tile_rows = a.tile_rows;
  p.max_tiles = a.max_tiles;
  p.out = a.out; p.out_stride = a.out_stride; p.route_weight = a.route_weight; p.permute_out = a.permute_out;
  p.status = a.status;
  p.gather_route = a.gather_route; p.gather_top_k = a.gather_top_k; p.gather_src = static_cast<const __nv_bfloat16*>(a.act);
  if (a.enc == ENC_Q4) return a.mode == 0 ? launch_wide<ENC_Q4, 0>(a, p, stream) : launch_wide<ENC_Q4, 1>(a, p, stream);
  if (a.enc == ENC_Q8) return a.mode == 0 ? launch_wide<ENC_Q8, 0>(a, p, stream) : launch_wide<ENC_Q8, 1>(a, p, stream);
  set_error("grouped: unknown encoding %d", a.enc);
  return ERR_BAD_ARGUMENT;
}

}  // namespace umaq
