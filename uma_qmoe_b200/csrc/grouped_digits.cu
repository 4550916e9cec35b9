// Grouped-expert GEMMs of Q8 layers on the int8 tensor cores, few routes per expert: D[weight row, route] = codes_e . digits^T.
//
// The activations come as two signed base-256 digits per value and one power-of-two scale per (row, 128 k) (digits.cuh), the
// weights stay the integers that they are stored as: the codes go from TMA to the tensor core without a conversion, which is
// what the BF16 kernels spend their time on while an expert has few routes.  A step of 128 k is one scale group of both
// operands: the tensor core forms the exact int32 sums of its products, and the epilogue warps add
// (256 * hi + lo) * weight scale * activation scale to float32 accumulators in registers.  No weight is rounded (the BF16
// kernels round code * scale to BF16): 2-norm of the error against 64 bits 0.0024 (of it 0.0023 the two roundings that every
// path has) against 0.0037.
//
//  * A tile is 256 weight rows (two M = 128 halves: gate and up rows of 128 features, or 256 down rows) x up to 64 routes;
//    N of an MMA is twice the routes (multiple of 16): rows [0, n) of the shared-memory tile are the upper digits, [n, 2n)
//    the lower ones.  128 features are one scale group of the down GEMM, so the gate/up epilogue leaves the SwiGLU result
//    (rounded to BF16, as everywhere) as digits itself.
//  * Tensor memory: a ring of four 128-column sums, one per half and step.
//  * One persistent CTA per SM: weight TMA (four stages of 32 KB), two warps copying the activation rows by index, MMA issuer,
//    eight epilogue warps (two groups of four, each taking half of the routes of both halves, so that a gate and its up
//    meet in a lane).
//  * The weight ring of the down GEMM starts to fill while the gate/up GEMM's last CTAs still run.
//
// Measured (B200, whole operator, us, transposed BF16 tiles | here): OLMoE 7 tokens 74 | 61, 96: 114 | 102, 192: 124 | 121;
// Qwen 24 tokens 128 | 96, 128: 142 | 119.  What bounds it: the last wave of tiles and a step of about 1700 clocks (1490 are
// its 34 KB of codes and scales).  Q4 codes as int8 operands (two words of 16 * code per word, through tensor memory) were slower
// than their BF16 conversion (7 tokens 53 | 70) and are not built.
#include "grouped.cuh"

#include <cuda.h>

#include "common.cuh"
#include "digits.cuh"
#include "tc.cuh"

namespace umaq {
namespace {

constexpr int kRows = 128;                // weight rows of a half = lanes of an MMA
constexpr int NMAX = kTileCapMin;         // routes of a tile
constexpr int kStepK = kDigitGroup;
constexpr int kDgMaxGroups = 16;          // K <= 2048
constexpr int kCopyThreads = 64;          // warps 2 and 3
constexpr int kEpilogueWarps = 8;
constexpr int kGroupThreads = kEpilogueWarps / 2 * 32;
constexpr int kUnitCols = 2 * NMAX;       // int32 sums of one half and step

constexpr int kHalfBytes = kRows * kStepK, kWeightBytes = 2 * kHalfBytes;
constexpr int kBTile = 2 * NMAX * kStepK;
constexpr int kPStages = 4, kBStages = 3, kUnits = 4;                  // 128 KB of codes in flight
constexpr int kDgTmemCols = kUnits * kUnitCols;
constexpr int kDgThreads = (4 + kEpilogueWarps) * 32;
static_assert(kDgTmemCols == 512, "tensor memory");

struct DgShared {
  uint64_t in_full[kBStages], in_empty[kBStages];
  uint64_t p_full[kPStages], p_empty[kPStages];
  uint64_t acc_full[kUnits], acc_empty[kUnits];
  uint64_t sc_full[2], sc_empty[2];                    // weight scales of a tile
  uint64_t sx_full[2], sx_empty[2];                    // activation scales of a tile
  uint32_t tmem_base;
  int abort_flag;
  int row[NMAX];                                       // the tile's activation rows
  uint32_t red[2][2][4][32];                           // [tile parity][group][lane quarter][route]: largest magnitudes
};

constexpr int kWeightScaleBytes = 2 * 2 * kRows * kDgMaxGroups * 4;
constexpr int kActScaleBytes = 2 * kDgMaxGroups * NMAX * 4;
constexpr size_t kDgSmemBytes = (size_t)kBStages * kBTile + (size_t)kPStages * kWeightBytes + kWeightScaleBytes + kActScaleBytes +
                                sizeof(DgShared) + 1024;
static_assert(kDgSmemBytes <= 227 * 1024, "shared memory of an SM");

// D (tensor memory, int32) += A x B of 32 int8 k, K-major operands in shared memory
__device__ __forceinline__ void tc_mma_i8(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// two float32 lanes per instruction
__device__ __forceinline__ uint64_t pack2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

struct DgTile {
  int col, expert, row0, nrows;
};
// The table is read through L2: the down GEMM's weight warp looks at it before its programmatic wait (see launch_dg).
__device__ __forceinline__ DgTile dg_tile(const GroupedParams& p, int it, int n_col) {
  DgTile t;
  const int m = it / n_col;
  t.col = it - m * n_col;
  t.expert = __ldcg(p.tile_expert + m); t.row0 = __ldcg(p.tile_row0 + m); t.nrows = __ldcg(p.tile_rows + m);
  return t;
}

template <int MODE>
__global__ void __launch_bounds__(kDgThreads, 1)
grouped_digits_kernel(const __grid_constant__ CUtensorMap map_w0, const __grid_constant__ CUtensorMap map_w1, const GroupedParams p) {
  constexpr int kFeatures = MODE == 0 ? kRows : 2 * kRows;                // output columns of a tile
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* sB = smem_raw;                                                 // [digit stages]
  uint8_t* sP = sB + kBStages * kBTile;                                // [code stages]
  float* sScales = reinterpret_cast<float*>(sP + kPStages * kWeightBytes);       // [2][256 rows][groups]
  float* sAct = sScales + kWeightScaleBytes / 4;                          // [2][groups][NMAX]
  DgShared& sh = *reinterpret_cast<DgShared*>(reinterpret_cast<uint8_t*>(sAct) + kActScaleBytes);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int K = p.k;
  const int nk = K / kStepK;                                              // steps = scale groups of a row
  const int n_col = p.n_rows / kFeatures;
  const int first = blockIdx.x, step = gridDim.x;
  volatile int* abort_flag = &sh.abort_flag;

  if (tid == 0) {
    for (int s = 0; s < kBStages; ++s) { mbar_init(&sh.in_full[s], kCopyThreads); mbar_init(&sh.in_empty[s], 1); }
    for (int s = 0; s < kPStages; ++s) { mbar_init(&sh.p_full[s], 1); mbar_init(&sh.p_empty[s], 1); }
    for (int s = 0; s < kUnits; ++s) { mbar_init(&sh.acc_full[s], 1); mbar_init(&sh.acc_empty[s], kEpilogueWarps); }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&sh.sc_full[s], 1); mbar_init(&sh.sc_empty[s], kEpilogueWarps);
      mbar_init(&sh.sx_full[s], kCopyThreads / 32); mbar_init(&sh.sx_empty[s], kEpilogueWarps);
    }
    sh.abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 0) {
    tmem_alloc(&sh.tmem_base, kDgTmemCols);
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
    Ring<kPStages> rp;
    Ring<kUnits> ru;
    uint32_t units = 0;
    const uint64_t b_desc0 = smem_desc_sw128(smem_u32(sB)), w_desc0 = smem_desc_sw128(smem_u32(sP));
    for (int it = first; it < total; it += step) {
      if (__any_sync(0xffffffffu, *abort_flag != 0)) break;
      const DgTile t = dg_tile(p, it, n_col);
      const int n16 = (t.nrows + 15) & ~15;
      // kind::i8, signed x signed -> int32, K-major operands, M = 128, N = two digits of the tile's routes
      const uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n16 >> 2) << 17) | (8u << 24);
      bool ok = true;
      for (int kc = 0; kc < nk; ++kc) {
        ok = ok && mbar_wait(&sh.in_full[rb.slot], rb.phase) && mbar_wait(&sh.p_full[rp.slot], rp.phase);
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          ok = ok && (units < (uint32_t)kUnits || mbar_wait(&sh.acc_empty[ru.slot], ru.phase ^ 1));
          if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
          tc_fence_after();
          if (half == 0) fence_proxy_async();
          if (elect_one()) {
            const uint64_t bd = b_desc0 + (uint64_t)(rb.slot * (kBTile >> 4));     // descriptors count 16-byte units
            const uint64_t wd = w_desc0 + (uint64_t)((rp.slot * kWeightBytes + half * kHalfBytes) >> 4);
            const uint32_t acc = tmem + ru.slot * kUnitCols;
#pragma unroll
            for (int k = 0; k < kStepK / 32; ++k) tc_mma_i8(acc, wd + k * 2, bd + k * 2, idesc, k ? 1u : 0u);
            tc_commit(&sh.acc_full[ru.slot]);
            if (half == 1) {
              tc_commit(&sh.p_empty[rp.slot]);
              tc_commit(&sh.in_empty[rb.slot]);
            }
          }
          __syncwarp();
          ru.next();
          ++units;
        }
        if (!ok) break;
        rb.next();
        rp.next();
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
        if (__any_sync(0xffffffffu, *abort_flag != 0)) break;
        const DgTile t = dg_tile(p, it, n_col);
        const long long wrow0 = (long long)t.expert * p.n_rows + t.col * kFeatures;
        const uint32_t sb = seq & 1;
        if (!__all_sync(0xffffffffu, seq < 2 || mbar_wait(&sh.sc_empty[sb], ((seq >> 1) - 1) & 1))) { if (lane == 0) fail(); break; }
        if (lane == 0) {
          float* dst_sc = sScales + sb * 2 * kRows * kDgMaxGroups;
          const uint32_t bytes = (uint32_t)kRows * nk * 4;
          mbar_expect_tx(&sh.sc_full[sb], 2 * bytes);
          bulk_g2s(dst_sc, p.scales0 + wrow0 * nk, bytes, &sh.sc_full[sb]);
          bulk_g2s(dst_sc + kRows * nk, MODE == 0 ? p.scales1 + wrow0 * nk : p.scales0 + (wrow0 + kRows) * nk, bytes, &sh.sc_full[sb]);
        }
        __syncwarp();
        ++seq;
        bool ok = true;
        for (int kc = 0; kc < nk; ++kc, ++kidx, rp.next()) {
          const uint32_t s = rp.slot;
          ok = __all_sync(0xffffffffu, kidx < (uint32_t)kPStages || mbar_wait(&sh.p_empty[s], rp.phase ^ 1));
          if (!ok) break;
          if (lane == 0) {
            mbar_expect_tx(&sh.p_full[s], kWeightBytes);
            uint8_t* dst = sP + s * kWeightBytes;
            tma_load_2d(dst, &map_w0, kc * kStepK, (int)wrow0, &sh.p_full[s]);
            if (MODE == 0) tma_load_2d(dst + kHalfBytes, &map_w1, kc * kStepK, (int)wrow0, &sh.p_full[s]);
            else tma_load_2d(dst + kHalfBytes, &map_w0, kc * kStepK, (int)wrow0 + kRows, &sh.p_full[s]);
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
  } else if (warp < 4) {
    // ===================== activation rows: 64 threads copy digits and scales by index ===========
    // A row of a step is 128 bytes of either digit = eight 16-byte chunks; chunk c of shared-memory row r lands at r * 128 +
    // ((c ^ (r & 7)) << 4), the 128-byte swizzle of the MMA descriptors.  Thread j copies chunk j & 7 of rows (j >> 3) + 8 i:
    // eight neighbouring lanes read one row's 128 contiguous bytes.  Rows up to the next multiple of 16 are zero-filled.
    const int pt = tid - 64;                              // 0 .. 63
    const int c = pt & 7, rbase = pt >> 3;
    const uint32_t dst_off = (uint32_t)rbase * 128 + (uint32_t)((c ^ rbase) << 4);
    const uint8_t* digits = reinterpret_cast<const uint8_t*>(p.gather_src) + c * 16;
    uint32_t kidx = 0, seq = 0;
    Ring<kBStages> rb;
    bool ok = true;
    for (int it = first; it < total; it += step, ++seq) {
      // everybody has read the previous tile's rows, and the threads agree whether to go on
      if (named_bar_or(1, kCopyThreads, !ok || *abort_flag != 0)) break;
      const DgTile t = dg_tile(p, it, n_col);
      const int n8 = ((t.nrows + 15) & ~15) >> 3;         // runs of 8 rows
      const uint32_t sb = seq & 1;
      int mine = -1;
      if (pt < t.nrows) mine = MODE == 0 ? p.gather_route[t.row0 + pt] / p.gather_top_k : t.row0 + pt;
      sh.row[pt] = mine;
      if (!__all_sync(0xffffffffu, seq < 2 || mbar_wait(&sh.sx_empty[sb], ((seq >> 1) - 1) & 1))) ok = false;
      float* sx = sAct + sb * kDgMaxGroups * NMAX + pt;
      const float* src_sx = p.act_scales + (size_t)(mine < 0 ? 0 : mine) * nk;
      for (int g = 0; g < nk; ++g) sx[g * NMAX] = mine < 0 ? 0.f : src_sx[g];
      __syncwarp();
      if (lane == 0) mbar_arrive(&sh.sx_full[sb]);
      named_bar_sync(1, kCopyThreads);
      int row[NMAX / 8];
#pragma unroll
      for (int i = 0; i < NMAX / 8; ++i) row[i] = sh.row[rbase + 8 * i];
      for (int kc = 0; kc < nk; ++kc, ++kidx, rb.next()) {
        if (!__all_sync(0xffffffffu, kidx < (uint32_t)kBStages || mbar_wait(&sh.in_empty[rb.slot], rb.phase ^ 1))) { ok = false; break; }
        uint8_t* dst = sB + rb.slot * kBTile + dst_off;
        const uint8_t* col = digits + kc * 2 * kStepK;
#pragma unroll
        for (int i = 0; i < NMAX / 8; ++i) {
          if (i < n8) {
            const uint8_t* src = col + (size_t)(row[i] < 0 ? 0 : row[i]) * K * 2;
            cp_async16(dst + i * 1024, src, row[i] >= 0);
            cp_async16(dst + (i + n8) * 1024, src + kStepK, row[i] >= 0);
          }
        }
        cp_async_arrive(&sh.in_full[rb.slot]);              // when they have landed; the issuer fences them towards the tensor core
      }
    }
    if (!ok && lane == 0) fail();
    cp_async_commit();
    cp_async_wait<0>();                                   // also on the abort path: nothing of this thread stays in flight
  } else {
    // ===================== epilogue warps: scaled sums in registers, then the result ==============
    // Lane = weight row of either half, column = route; group g of four warps takes routes [g * n / 2, (g + 1) * n / 2).
    const int group = (warp - 4) >> 2, quarter = warp & 3;
    const int row = quarter * 32 + lane;
    const uint32_t lane_base = tmem + ((uint32_t)(quarter * 32) << 16);
    const bool vec = (nk & 3) == 0;
    uint32_t seq = 0;
    Ring<kUnits> ru;
    bool ok = true;
    for (int it = first; it < total; it += step, ++seq) {
      if (MODE == 1 && *abort_flag) break;
      const DgTile t = dg_tile(p, it, n_col);
      const int n16 = (t.nrows + 15) & ~15, half_n = n16 >> 1, chunks = n16 >> 4;     // 8-route chunks of this group
      const uint32_t sb = seq & 1;
      ok = ok && mbar_wait(&sh.sc_full[sb], (seq >> 1) & 1) && mbar_wait(&sh.sx_full[sb], (seq >> 1) & 1);
      const float* sw = sScales + sb * 2 * kRows * kDgMaxGroups + row * nk;
      const float* sx = sAct + sb * kDgMaxGroups * NMAX + group * half_n;
      uint64_t acc[2][NMAX / 4];
#pragma unroll
      for (int i = 0; i < NMAX / 4; ++i) acc[0][i] = acc[1][i] = 0;
      float4 s4[2];
      for (int kc = 0; kc < nk && ok; ++kc, sx += NMAX) {
        const int j = kc & 3;
        if (vec) {                                          // rows 64 bytes apart: four scales per load, a quarter of the conflicts
          if (j == 0) {
            s4[0] = *reinterpret_cast<const float4*>(sw + kc);
            s4[1] = *reinterpret_cast<const float4*>(sw + kRows * nk + kc);
          }
        } else {
          s4[0].x = s4[0].y = s4[0].z = s4[0].w = sw[kc];
          s4[1].x = s4[1].y = s4[1].z = s4[1].w = sw[kRows * nk + kc];
        }
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const float s = j < 2 ? (j == 0 ? s4[half].x : s4[half].y) : (j == 2 ? s4[half].z : s4[half].w);
          const uint64_t s2 = pack2(s, s);
          ok = ok && mbar_wait(&sh.acc_full[ru.slot], ru.phase);
          if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
          tc_fence_after();
          const uint32_t base = lane_base + ru.slot * kUnitCols + group * half_n;
          uint32_t hi[2][8], lo[2][8];
          tmem_ld8(base, hi[0]);
          tmem_ld8(base + n16, lo[0]);
#pragma unroll
          for (int c = 0; c < NMAX / 16; ++c) {
            if (c < chunks) {
              tmem_ld_wait();
              if (c + 1 < chunks) {                         // the next chunk's reads run under this one's arithmetic
                tmem_ld8(base + (c + 1) * 8, hi[(c + 1) & 1]);
                tmem_ld8(base + n16 + (c + 1) * 8, lo[(c + 1) & 1]);
              } else {
                tc_fence_before();                          // every tcgen05.ld of this sum is complete (wait::ld)
                __syncwarp();
                if (lane == 0) mbar_arrive(&sh.acc_empty[ru.slot]);
              }
              const ulonglong2 x01 = *reinterpret_cast<const ulonglong2*>(sx + c * 8);
              const ulonglong2 x23 = *reinterpret_cast<const ulonglong2*>(sx + c * 8 + 4);
              const uint64_t xs[4] = {x01.x, x01.y, x23.x, x23.y};
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                // |sum| < 2^30: 128 products of a code and a 16-bit integer
                const int d0 = ((int)hi[c & 1][2 * i] << 8) + (int)lo[c & 1][2 * i];
                const int d1 = ((int)hi[c & 1][2 * i + 1] << 8) + (int)lo[c & 1][2 * i + 1];
                acc[half][c * 4 + i] = fma2(pack2(__int2float_rn(d0), __int2float_rn(d1)), mul2(xs[i], s2), acc[half][c * 4 + i]);
              }
            }
          }
          ru.next();
        }
      }
      __syncwarp();
      if (lane == 0) { mbar_arrive(&sh.sc_empty[sb]); mbar_arrive(&sh.sx_empty[sb]); }
      const int route0 = group * half_n;                    // this group's first route of the tile
      const int left = min(half_n, t.nrows - route0);       // its routes (none, if <= 0)
      if (MODE == 0) {
        // SwiGLU, rounded to BF16; the largest magnitude of each route over the tile's 128 features; digits
        uint32_t top = 0;                                   // lane j: route j's largest magnitude among this warp's features
#pragma unroll
        for (int i = 0; i < NMAX / 4; ++i) {
          if (2 * i < half_n) {
            float g0, g1, u0, u1;
            unpack2(acc[0][i], g0, g1);
            unpack2(acc[1][i], u0, u1);
            g0 = bf16_round(silu_f32(g0) * u0);
            g1 = bf16_round(silu_f32(g1) * u1);
            const uint32_t m0 = __reduce_max_sync(0xffffffffu, __float_as_uint(g0) & 0x7fffffffu);
            const uint32_t m1 = __reduce_max_sync(0xffffffffu, __float_as_uint(g1) & 0x7fffffffu);
            if (lane == 2 * i) top = m0;
            if (lane == 2 * i + 1) top = m1;
            acc[0][i] = pack2(g0, g1);
          }
        }
        uint32_t (*red)[32] = sh.red[sb][group];            // by tile parity: a warp is at most one tile ahead of its group
        red[quarter][lane] = top;
        if (named_bar_or(2 + group, kGroupThreads, !ok || *abort_flag != 0)) { ok = false; break; }
        top = max(max(red[0][lane], red[1][lane]), max(red[2][lane], red[3][lane]));
        const DigitScale ds = digit_scale(top);
        const long long r0 = (long long)t.row0 + route0;
        if (quarter == 0 && lane < left) p.out_scales[(r0 + lane) * (p.n_rows / kDigitGroup) + t.col] = ds.to_value;
        uint8_t* dst = reinterpret_cast<uint8_t*>(p.out) + r0 * 2 * p.n_rows + t.col * 2 * kDigitGroup + row;
#pragma unroll
        for (int i = 0; i < NMAX / 4; ++i) {
          if (2 * i < left) {
            float h[2];
            unpack2(acc[0][i], h[0], h[1]);
#pragma unroll
            for (int o = 0; o < 2; ++o) {
              const float f = __shfl_sync(0xffffffffu, ds.to_int, 2 * i + o);
              if (2 * i + o < left) {
                int q1, q0;
                to_digits(h[o], f, q1, q0);
                uint8_t* at = dst + (long long)(2 * i + o) * 2 * p.n_rows;
                at[0] = (uint8_t)q1;
                at[kDigitGroup] = (uint8_t)q0;
              }
            }
          }
        }
      } else {
        if (!ok) break;
        const float wr = lane < left ? p.route_weight[t.row0 + route0 + lane] : 0.f;
        __nv_bfloat16* dst = p.out + ((long long)t.row0 + route0) * p.out_stride + t.col * kFeatures + row;
#pragma unroll
        for (int i = 0; i < NMAX / 4; ++i) {
          if (2 * i < left) {
            const float w0 = __shfl_sync(0xffffffffu, wr, 2 * i), w1 = __shfl_sync(0xffffffffu, wr, 2 * i + 1);
#pragma unroll
            for (int half = 0; half < 2; ++half) {
              float y0, y1;
              unpack2(acc[half][i], y0, y1);
              __nv_bfloat16* at = dst + (long long)(2 * i) * p.out_stride + half * kRows;
              at[0] = __float2bfloat16_rn(y0 * w0);
              if (2 * i + 1 < left) at[p.out_stride] = __float2bfloat16_rn(y1 * w1);
            }
          }
        }
      }
    }
    if (!ok && lane == 0) fail();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem, kDgTmemCols);
  }
}

template <int MODE>
int launch_dg(const GroupedGemmArgs& a, const GroupedParams& p, cudaStream_t stream) {
  auto kernel = grouped_digits_kernel<MODE>;
  static thread_local int configured = -1;
  int dev = 0;
  cudaGetDevice(&dev);
  if (configured != dev) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDgSmemBytes);
    if (e != cudaSuccess) { set_error("grouped: cudaFuncSetAttribute: %s", cudaGetErrorString(e)); return ERR_LAUNCH; }
    configured = dev;
  }
  CUtensorMap m0, m1;
  const uint64_t wrows = (uint64_t)a.num_experts * a.n_rows, rowb = a.k;
  if (!make_map(&m0, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, a.w0, rowb, wrows, kStepK, kRows, CU_TENSOR_MAP_SWIZZLE_128B) ||
      !make_map(&m1, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, MODE == 0 ? a.w1 : a.w0, rowb, wrows, kStepK, kRows, CU_TENSOR_MAP_SWIZZLE_128B))
    return ERR_LAUNCH;
  const cudaError_t e = launch_chained(kernel, dim3(sm_count()), dim3(kDgThreads), kDgSmemBytes, stream, m0, m1, p);
  if (e != cudaSuccess) { set_error("grouped: launch failed: %s", cudaGetErrorString(e)); return ERR_LAUNCH; }
  return ERR_NONE;
}

}  // namespace

// Both GEMMs of a layer, the down GEMM directly behind the gate/up GEMM on the stream (its weight warp relies on it).
int launch_grouped_gemm_digits(const GroupedGemmArgs& a, cudaStream_t stream) {
  if (a.enc != ENC_Q8 || a.k % kStepK || a.k > kDgMaxGroups * kStepK || a.n_rows % (a.mode == 0 ? kRows : 2 * kRows) || a.total_rows <= 0 ||
      a.max_tiles <= 0 || a.tile_cap > NMAX || !a.act_scales || (a.mode == 0 ? !a.gather_route || a.gather_top_k < 1 || !a.out_scales : !a.route_weight)) {
    set_error("grouped: unsupported shape (k %d, rows per expert %d)", a.k, a.n_rows);
    return ERR_BAD_ARGUMENT;
  }
  GroupedParams p{};
  p.k = a.k; p.n_rows = a.n_rows;
  p.scales0 = a.s0; p.scales1 = a.s1;
  p.num_tiles = a.num_tiles; p.tile_expert = a.tile_expert; p.tile_row0 = a.tile_row0; p.tile_rows = a.tile_rows;
  p.max_tiles = a.max_tiles;
  p.out = a.out; p.out_stride = a.out_stride; p.out_scales = a.out_scales; p.route_weight = a.route_weight;
  p.status = a.status;
  p.gather_route = a.gather_route; p.gather_top_k = a.gather_top_k; p.gather_src = static_cast<const __nv_bfloat16*>(a.act);
  p.act_scales = a.act_scales;
  return a.mode == 0 ? launch_dg<0>(a, p, stream) : launch_dg<1>(a, p, stream);
}

}  // namespace umaq
