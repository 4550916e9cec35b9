// Grouped-expert GEMMs with the weights as the M operand: D[weight row, route] = W_e . x^T.
//
// Same contract as grouped.cu (gate/up + SwiGLU, down x routing weight, over routes sorted by expert; replaces
// src/uma_qmoe/native/packed_q4_kernel.cu:560-776, :894-1099), transposed:
//
//  * 128 weight rows are the 128 lanes of one tcgen05.mma and the routes are its N (a multiple of 16).  The tensor time
//    of a tile follows the routes it has, instead of 128 or 256 of them being multiplied for every expert.
//  * The converted weights are the A operand in TENSOR MEMORY: a conversion thread owns one weight row = one lane, turns
//    its packed codes into BF16 words and stores them with tcgen05.st, with no pass through shared memory and no proxy fence.
//
// A tile is 128 weight rows x up to 64 routes; two CTAs per SM, accumulators double-buffered (2 x 64 columns) beside the
// converted weights.  For experts with few routes the bound is the stream of packed weights; two independent CTAs with
// separate epilogue warps keep it going.  Gate and up rows share the 128 lanes (16 and 16 in every lane quarter).
//
// BF16 layers need no conversion: TMA writes the swizzled A tile to shared memory.
//
// Measured (B200, OLMoE shape, 64 tokens = 8 routes per expert, gate/up | down, us; the kernels of grouped.cu in brackets):
// Q4 46 | 27 (106 | 58), Q8 71 | 38 (138 | 71) = 4.0 TB/s of codes.  What bounds the quantised encodings is the conversion:
// of 1850 clocks a 128-k step takes a CTA, 760 (Q4) are its arithmetic, 460 its loop, 160 the tcgen05.st.  With 64-k steps
// and a lone lane computing descriptors the MMA issuer was the bound (1200 clocks a step for four MMAs): 54 | 29.  Qwen BF16,
// 512 tokens: 126 | 61 (132 | 70), gate/up at 0.83 of the copy bandwidth.
//
// K order as in grouped.cu: the quantised paths use [k0,k4,k1,k5,k2,k6,k3,k7] inside every run of 8 k, for both operands.
#include "grouped.cuh"

#include <cuda.h>

#include "common.cuh"
#include "tc.cuh"

namespace umaq {
namespace {

constexpr int kRows = 128;                // weight rows of a tile = lanes of the MMA
constexpr int NMAX = 64;                  // routes of a tile
constexpr int kAtomK = 64;                // k of one 128-byte swizzle atom of BF16
constexpr int kActBox = 16;               // rows of an activation TMA box
constexpr int kTsMaxGroups = 16;          // quantised K <= 2048
constexpr int kAccBufs = 2;
constexpr int kTsGatherThreads = 64;      // warps 2 and 3 when the activation rows are fetched by index
constexpr int kEpilogueWarps = 4;

// A step is 128 k (one scale group) for the quantised encodings: the waits, commits and index arithmetic of a step cost the
// issuing and the converting warps as much as its work at 64 k.  BF16 steps are 64 k (16 KB of weights).
template <int ENC>
struct TsShape {
  static constexpr bool kQuant = ENC != ENC_BF16;
  static constexpr int kAtoms = kQuant ? 2 : 1;
  static constexpr int kStepK = kAtoms * kAtomK;
  static constexpr int kPackedRow = ENC == ENC_Q4 ? kStepK / 2 : kStepK;   // code bytes of a row and step
  static constexpr int kWeightBytes = kRows * (kQuant ? kPackedRow : kStepK * 2);
  static constexpr int kBAtom = NMAX * 128;                                // activation tile, one atom
  static constexpr int kBTile = kAtoms * kBAtom;
  static constexpr int kPStages = ENC == ENC_Q4 ? 4 : ENC == ENC_Q8 ? 3 : 4;
  static constexpr int kBStages = ENC == ENC_Q4 ? 3 : ENC == ENC_Q8 ? 2 : 4;   // what 113 KB hold beside the codes
  static constexpr int kAccCols = kAccBufs * NMAX;
  static constexpr int kAStages = kQuant ? 2 : 1;                          // BF16: no ring, one unused pair of barriers
  static constexpr int kTmemCols = kQuant ? 256 : 128;
  static constexpr int kConvertWarps = kQuant ? 8 : 0;
  static constexpr int kThreads = (4 + kConvertWarps + kEpilogueWarps) * 32;
  static constexpr int kScaleBytes = kQuant ? 2 * kRows * kTsMaxGroups * 4 : 0;
  static_assert(kAccCols + (kQuant ? kAStages * kStepK / 2 : 0) <= kTmemCols, "tensor memory");
};

template <int ENC>
struct TsShared {
  using S = TsShape<ENC>;
  uint64_t in_full[S::kBStages], in_empty[S::kBStages];
  uint64_t p_full[S::kPStages], p_empty[S::kPStages];
  uint64_t a_full[S::kAStages], a_empty[S::kAStages];
  uint64_t sc_full[2], sc_empty[2];
  uint64_t acc_full[kAccBufs], acc_empty[kAccBufs];
  uint32_t tmem_base;
  int abort_flag;
  int gather_token[NMAX];
};

template <int ENC>
constexpr size_t ts_smem_bytes() {
  using S = TsShape<ENC>;
  return (size_t)S::kBStages * S::kBTile + (size_t)S::kPStages * S::kWeightBytes + S::kScaleBytes + sizeof(TsShared<ENC>) + 1024;
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}

struct TsTile {
  int col, expert, row0, nrows;
  int part, k0, k1;                         // part of the contraction, its first and end step
};

// tile table entry -> one of its `subs` parts of at most NMAX routes (equal parts, multiples of 16); nrows 0: no such part.
// WIDE: entries may have more than NMAX routes (a table cut for the other kernels).  A template parameter, since the branch
// costs every role of every tile 2 % of a small batch.
template <bool SPLIT, bool WIDE>
__device__ __forceinline__ TsTile ts_tile(const GroupedParams& p, int it, int n_col, int nk) {
  TsTile t;
  t.part = 0; t.k0 = 0; t.k1 = nk;
  if (SPLIT && p.k_splits > 1) {
    const int each = (nk + p.k_splits - 1) / p.k_splits;
    t.part = it % p.k_splits;
    it /= p.k_splits;
    t.k0 = min(nk, t.part * each); t.k1 = min(nk, t.k0 + each);
  }
  const int m = it / n_col;
  t.col = it - m * n_col;
  // Many experts: every entry's first part, then every entry's second one.  A dense matrix, whose entries are full: entry by
  // entry.  Either way the parts that exist come one after another and spread evenly over the CTAs.
  int sub = 0, tm = m;
  if (WIDE) {
    if (p.part_major) {
      const int entries = *p.num_tiles;
      sub = m / entries; tm = m - sub * entries;
    } else {
      tm = m / p.subs; sub = m - tm * p.subs;
    }
  }
  t.expert = p.tile_expert[tm]; t.row0 = p.tile_row0[tm]; t.nrows = p.tile_rows[tm];
  if (WIDE) {
    const int parts = (t.nrows + NMAX - 1) / NMAX;
    const int each = ((t.nrows + parts - 1) / parts + 15) & ~15;
    t.row0 += sub * each;
    t.nrows = max(0, min(each, t.nrows - sub * each));
  }
  return t;
}

template <int ENC, int MODE, bool WIDE>
__global__ void __launch_bounds__(TsShape<ENC>::kThreads, 2)
grouped_ts_kernel(const __grid_constant__ CUtensorMap map_act, const __grid_constant__ CUtensorMap map_w0,
                  const __grid_constant__ CUtensorMap map_w1, const GroupedParams p) {
  using S = TsShape<ENC>;
  constexpr bool kQuant = S::kQuant;
  constexpr int kPStages = S::kPStages, kBStages = S::kBStages, kAStages = S::kAStages;
  constexpr int kFeatures = MODE == 0 ? kRows / 2 : kRows;                // output columns of a tile
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* sB = smem_raw;                                                 // [activation stages]
  uint8_t* sP = sB + kBStages * S::kBTile;                                // [weight stages: codes, or BF16 A tiles]
  float* sScales = reinterpret_cast<float*>(sP + kPStages * S::kWeightBytes);
  TsShared<ENC>& sh = *reinterpret_cast<TsShared<ENC>*>(reinterpret_cast<uint8_t*>(sScales) + S::kScaleBytes);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int K = p.k;
  const int nk = K / S::kStepK;
  const int groups = K >> 7;
  const int n_col = p.n_rows / kFeatures;
  constexpr bool kSplit = !kQuant && MODE == 1;
  const int first = blockIdx.x, step = gridDim.x;
  volatile int* abort_flag = &sh.abort_flag;
  const bool gather = MODE == 0 && p.gather_route != nullptr;

  pdl_launch_dependents();
  if (p.conditional && !launch_runs(p)) return;                        // an ordinary launch: what it reads here was written before
  if (tid == 0) {
    for (int s = 0; s < kBStages; ++s) { mbar_init(&sh.in_full[s], gather ? kTsGatherThreads : 1); mbar_init(&sh.in_empty[s], 1); }
    for (int s = 0; s < kPStages; ++s) { mbar_init(&sh.p_full[s], 1); mbar_init(&sh.p_empty[s], kQuant ? S::kConvertWarps : 1); }
    for (int s = 0; s < kAStages; ++s) { mbar_init(&sh.a_full[s], kQuant ? S::kConvertWarps : 1); mbar_init(&sh.a_empty[s], 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(&sh.sc_full[s], 1); mbar_init(&sh.sc_empty[s], kQuant ? S::kConvertWarps : 1); }
    for (int s = 0; s < kAccBufs; ++s) { mbar_init(&sh.acc_full[s], 1); mbar_init(&sh.acc_empty[s], kEpilogueWarps); }
    sh.abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 0) {
    tmem_alloc(&sh.tmem_base, S::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sh.tmem_base;
  const int total = *p.num_tiles * (WIDE ? p.subs : 1) * n_col * (kSplit ? p.k_splits : 1);
  auto fail = [&]() { atomicExch(p.status, (unsigned)ERR_DEVICE_TIMEOUT); *abort_flag = 1; };

  if (warp == 0) {
    // ===================== MMA issuer: the warp stays converged, one elected lane issues ==========
    Ring<kBStages> rb;
    Ring<kAStages> ra;
    Ring<kPStages> rp;
    const uint64_t b_desc0 = smem_desc_sw128(smem_u32(sB)), w_desc0 = smem_desc_sw128(smem_u32(sP));
    uint32_t seq = 0;
    for (int it = first; it < total; it += step) {
      if (warp_sees(abort_flag)) break;
      const TsTile t = ts_tile<kSplit, WIDE>(p, it, n_col, nk);
      if (t.nrows == 0) continue;
      const uint32_t buf = seq % kAccBufs, use = seq / kAccBufs;
      ++seq;
      bool ok = use == 0 || mbar_wait_warp(&sh.acc_empty[buf], (use - 1) & 1);
      const int n16 = (t.nrows + 15) & ~15;
      // kind::f16, BF16 x BF16 -> FP32, K-major operands, M = 128, N = the tile's routes
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n16 >> 3) << 17) | (8u << 24);
      const uint32_t acc = tmem + buf * NMAX;
      for (int kc = t.k0; kc < t.k1; ++kc) {
        ok = __all_sync(0xffffffffu, ok && mbar_wait(&sh.in_full[rb.slot], rb.phase) &&
                                         (kQuant ? mbar_wait(&sh.a_full[ra.slot], ra.phase) : mbar_wait(&sh.p_full[rp.slot], rp.phase)));
        if (!ok) break;
        tc_fence_after();
        if (gather) fence_proxy_async();
        if (elect_one()) {
          const uint64_t bd = b_desc0 + (uint64_t)(rb.slot * (S::kBTile >> 4));       // descriptors count 16-byte units
          const uint64_t wd = w_desc0 + (uint64_t)(rp.slot * (S::kWeightBytes >> 4));
          const uint32_t a_tmem = tmem + S::kAccCols + ra.slot * (S::kStepK / 2);
#pragma unroll
          for (int k = 0; k < S::kStepK / 16; ++k) {
            const uint64_t bdesc = bd + (k >> 2) * (S::kBAtom >> 4) + (k & 3) * 2;
            const uint32_t accumulate = k ? 1u : (uint32_t)(kc != t.k0);
            if (kQuant) tc_mma_bf16_ts(acc, a_tmem + k * 8, bdesc, idesc, accumulate);
            else tc_mma_bf16(acc, wd + k * 2, bdesc, idesc, accumulate);
          }
          tc_commit(kQuant ? &sh.a_empty[ra.slot] : &sh.p_empty[rp.slot]);
          tc_commit(&sh.in_empty[rb.slot]);
          if (kc == t.k1 - 1) tc_commit(&sh.acc_full[buf]);
        }
        __syncwarp();
        rb.next();
        if (kQuant) ra.next(); else rp.next();
      }
      if (!ok) { if (lane == 0) fail(); break; }
    }
  } else if (warp == 1) {
    // ===================== TMA producer: scales and weight rows ==================================
    // The whole warp waits (a lone lane's wait takes twice as long and slows the others'), one lane issues.
    {
      uint32_t kidx = 0, seq = 0;
      Ring<kPStages> rp;
      for (int it = first; it < total; it += step) {
        if (warp_sees(abort_flag)) break;
        const TsTile t = ts_tile<kSplit, WIDE>(p, it, n_col, nk);
        if (t.nrows == 0) continue;
        const long long wrow0 = (long long)t.expert * p.n_rows + t.col * kFeatures;
        if (kQuant) {
          const uint32_t sb = seq & 1;
          if (!__all_sync(0xffffffffu, seq < 2 || mbar_wait(&sh.sc_empty[sb], ((seq >> 1) - 1) & 1))) { if (lane == 0) fail(); break; }
          float* dst = sScales + sb * kRows * kTsMaxGroups;
          const uint32_t bytes = (uint32_t)kFeatures * groups * 4;
          if (lane == 0) {
            mbar_expect_tx(&sh.sc_full[sb], MODE == 0 ? 2 * bytes : bytes);
            bulk_g2s(dst, p.scales0 + wrow0 * groups, bytes, &sh.sc_full[sb]);
            if (MODE == 0) bulk_g2s(dst + kFeatures * groups, p.scales1 + wrow0 * groups, bytes, &sh.sc_full[sb]);
          }
          __syncwarp();
        }
        ++seq;
        bool ok = true;
        for (int kc = t.k0; kc < t.k1; ++kc, ++kidx, rp.next()) {
          const uint32_t s = rp.slot;
          ok = __all_sync(0xffffffffu, kidx < (uint32_t)kPStages || mbar_wait(&sh.p_empty[s], rp.phase ^ 1));
          if (!ok) break;
          if (lane == 0) mbar_expect_tx(&sh.p_full[s], S::kWeightBytes);
          __syncwarp();
          uint8_t* dst = sP + s * S::kWeightBytes;
          if (!kQuant && MODE == 0) {
            // 16 gate rows and the 16 up rows of the same features share a lane quarter: boxes of 16 rows, a lane each
            if (lane < 8)
              tma_load_2d(dst + lane * 16 * 128, lane & 1 ? &map_w1 : &map_w0, kc * kAtomK, (int)wrow0 + (lane >> 1) * 16, &sh.p_full[s]);
          } else if (lane != 0) {
          } else if (kQuant) {
            tma_load_2d(dst, &map_w0, kc * S::kPackedRow, (int)wrow0, &sh.p_full[s]);
            if (MODE == 0) tma_load_2d(dst + kFeatures * S::kPackedRow, &map_w1, kc * S::kPackedRow, (int)wrow0, &sh.p_full[s]);
          } else {
            tma_load_2d(dst, &map_w0, kc * kAtomK, (int)wrow0, &sh.p_full[s]);
          }
          __syncwarp();
        }
        if (!ok) { if (lane == 0) fail(); break; }
      }
      if (*abort_flag) {                                // nobody consumes: wait (bounded) for the copies in flight
        if (kQuant)
          for (uint32_t q = seq > 2 ? seq - 2 : 0; q < seq; ++q) mbar_wait(&sh.sc_full[q & 1], (q >> 1) & 1);
        for (uint32_t k2 = kidx > (uint32_t)kPStages ? kidx - kPStages : 0; k2 < kidx; ++k2)
          mbar_wait(&sh.p_full[k2 % kPStages], (k2 / kPStages) & 1);
      }
    }
  } else if (warp < 4) {
    if (!gather) {
      // ===================== TMA producer: activation rows in sorted order =========================
      if (warp == 2) {
        uint32_t kidx = 0;
        Ring<kBStages> rb;
        for (int it = first; it < total; it += step) {
          if (warp_sees(abort_flag)) break;
          const TsTile t = ts_tile<kSplit, WIDE>(p, it, n_col, nk);
          if (t.nrows == 0) continue;
          const int boxes = (t.nrows + kActBox - 1) / kActBox;
          bool ok = true;
          for (int kc = t.k0; kc < t.k1; ++kc, ++kidx, rb.next()) {
            const uint32_t s = rb.slot;
            ok = __all_sync(0xffffffffu, kidx < (uint32_t)kBStages || mbar_wait(&sh.in_empty[s], rb.phase ^ 1));
            if (!ok) break;
            if (lane == 0) mbar_expect_tx(&sh.in_full[s], S::kAtoms * boxes * kActBox * 128);
            __syncwarp();
            if (lane < S::kAtoms * boxes) {                 // a box per lane
              const int a = lane / boxes, b = lane - a * boxes;
              tma_load_2d(sB + s * S::kBTile + a * S::kBAtom + b * kActBox * 128, &map_act, kc * S::kStepK + a * kAtomK,
                          t.row0 + b * kActBox, &sh.in_full[s]);
            }
            __syncwarp();
          }
          if (!ok) { if (lane == 0) fail(); break; }
        }
        if (*abort_flag)
          for (uint32_t k2 = kidx > (uint32_t)kBStages ? kidx - kBStages : 0; k2 < kidx; ++k2)
            mbar_wait(&sh.in_full[k2 % kBStages], (k2 / kBStages) & 1);
      }
    } else {
      // ===================== gather producers: 64 threads write every activation tile ===============
      // As in grouped.cu: thread j copies 16-byte chunk j & 7 (of each atom) of rows (j >> 3) + 8 i into the 128-byte-
      // swizzled slot, so eight neighbouring lanes read one row's 128 contiguous bytes.  Rows up to the next multiple of
      // 16 are zero-filled.
      const int pt = tid - 64;                              // 0 .. 63
      const int c = pt & 7, rbase = pt >> 3;                // rows rbase + 8 i: all have r & 7 == rbase
      const uint32_t dst_off = (uint32_t)rbase * 128 + (uint32_t)((c ^ rbase) << 4);
      uint32_t kidx = 0;
      Ring<kBStages> rb;
      bool ok = true;
      for (int it = first; it < total; it += step) {
        // everybody has read the previous tile's table, and the threads agree whether to go on
        if (named_bar_or(1, kTsGatherThreads, !ok || *abort_flag != 0)) break;
        const TsTile t = ts_tile<kSplit, WIDE>(p, it, n_col, nk);
        const int n8 = ((t.nrows + 15) & ~15) >> 3;         // runs of 8 rows
        sh.gather_token[pt] = pt < t.nrows ? p.gather_route[t.row0 + pt] / p.gather_top_k : -1;
        named_bar_sync(1, kTsGatherThreads);
        if (t.nrows == 0) continue;
        int tok[NMAX / 8];
#pragma unroll
        for (int i = 0; i < NMAX / 8; ++i) tok[i] = sh.gather_token[rbase + 8 * i];
        const uint8_t* col = reinterpret_cast<const uint8_t*>(p.gather_src) + c * 16;
        for (int kc = 0; kc < nk; ++kc, ++kidx, rb.next(), col += S::kStepK * 2) {
          if (!__all_sync(0xffffffffu, kidx < (uint32_t)kBStages || mbar_wait(&sh.in_empty[rb.slot], rb.phase ^ 1))) { ok = false; break; }
          uint8_t* dst = sB + rb.slot * S::kBTile + dst_off;
#pragma unroll
          for (int i = 0; i < NMAX / 8; ++i) {
            if (i < n8) {
              const uint8_t* src = col + (size_t)(tok[i] < 0 ? 0 : tok[i]) * K * 2;
#pragma unroll
              for (int a = 0; a < S::kAtoms; ++a) cp_async16(dst + a * S::kBAtom + i * 1024, src + a * 128, tok[i] >= 0);
            }
          }
          cp_async_arrive(&sh.in_full[rb.slot]);            // when they have landed; the issuer fences them towards the tensor core
        }
      }
      if (!ok && lane == 0) fail();
      cp_async_commit();
      cp_async_wait<0>();                                   // also on the abort path: nothing of this thread stays in flight
    }
  } else if (kQuant && warp < 4 + S::kConvertWarps) {
    // ===================== conversion warps: packed codes -> BF16 rows of A in tensor memory =========
    // A thread owns one row = one lane; the two warpgroups take the two 64-k atoms of a step.
    const int quarter = warp & 3, half = (warp - 4) >> 2;
    const int row = MODE == 0 ? (lane < 16 ? 0 : 64) + quarter * 16 + (lane & 15)   // lanes 0-15 gate, 16-31 up
                              : quarter * 32 + lane;
    const uint32_t a_lane = tmem + ((uint32_t)(quarter * 32) << 16) + S::kAccCols + half * 32;
    uint32_t kidx = 0, seq = 0;
    Ring<kPStages> rp;
    Ring<kAStages> ra;
    for (int it = first; it < total; it += step) {
      const TsTile t = ts_tile<kSplit, WIDE>(p, it, n_col, nk);
      if (t.nrows == 0) continue;
      const uint32_t sbuf = seq & 1;
      mbar_wait_or_flag(&sh.sc_full[sbuf], (seq >> 1) & 1, abort_flag);
      ++seq;
      const float* sc = sScales + sbuf * kRows * kTsMaxGroups + row * groups;
      for (int kc = 0; kc < nk; ++kc, ++kidx) {
        const float scale = sc[kc];
        const Q4Scale qs = q4_scale(scale);
        const bool fused = ENC == ENC_Q4 && __all_sync(0xffffffffu, qs.fused);
        mbar_wait_or_flag(&sh.p_full[rp.slot], rp.phase, abort_flag);
        const uint8_t* src = sP + rp.slot * S::kWeightBytes + row * S::kPackedRow;
        uint32_t out[2][16];
#pragma unroll
        for (int j = 0; j < 2; ++j) {                       // 32 codes each
          if (ENC == ENC_Q4) {                              // 64-byte rows, TMA swizzle: 16-byte chunk ^ (row >> 1 & 3)
            const uint4 raw = *reinterpret_cast<const uint4*>(src + (((2 * half + j) ^ ((row >> 1) & 3)) << 4));
            if (fused) convert_q4_fused(raw, qs, out[j]);
            else convert_q4(raw, scale, out[j]);
          } else {                                          // 128-byte rows: chunk ^ (row & 7)
            const int c = 4 * half + 2 * j;
            convert_q8(*reinterpret_cast<const uint4*>(src + ((c ^ (row & 7)) << 4)),
                       *reinterpret_cast<const uint4*>(src + (((c + 1) ^ (row & 7)) << 4)), scale, out[j]);
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh.p_empty[rp.slot]);
        if (kidx >= (uint32_t)kAStages) mbar_wait_or_flag(&sh.a_empty[ra.slot], ra.phase ^ 1, abort_flag);
        tc_fence_after();
#pragma unroll
        for (int j = 0; j < 2; ++j) tmem_st16(a_lane + ra.slot * (S::kStepK / 2) + j * 16, out[j]);
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
    // Lane = weight row, column = route.  Neighbouring output columns sit in neighbouring lanes, so pairs of lanes swap
    // one route of each pair of routes and a store instruction writes 4-byte words of two (four) rows.
    const int quarter = warp & 3;
    const uint32_t lane_base = tmem + ((uint32_t)(quarter * 32) << 16);
    uint32_t seq = 0;
    for (int it = first; it < total; it += step) {
      const TsTile t = ts_tile<kSplit, WIDE>(p, it, n_col, nk);
      if (t.nrows == 0) continue;
      const uint32_t buf = seq % kAccBufs, use = seq / kAccBufs;
      ++seq;
      if (!mbar_wait_warp(&sh.acc_full[buf], use & 1) || warp_sees(abort_flag)) { if (lane == 0) fail(); break; }
      tc_fence_after();
      const int chunks = (t.nrows + 15) >> 4;
      const uint32_t acc = lane_base + buf * NMAX;
      for (int c = 0; c < chunks; ++c) {
        const int left = t.nrows - c * 16;                  // routes of this chunk
        __nv_bfloat16* orow = p.out + ((long long)t.row0 + c * 16) * p.out_stride + t.col * kFeatures;
        uint32_t a[16];
        tmem_ld16(acc + c * 16, a);
        tmem_ld_wait();
        if (MODE == 0) {
          // lanes 0-15 hold gate rows, lanes 16-31 the up rows of the same 16 features: each half takes one route of a pair
          const bool up = lane >= 16;
          const int f = lane & 15;
          const int hi = p.permute_out ? (f >> 2) & 1 : f & 1;
          const int swap = p.permute_out ? 4 : 1;
          // word of an 8-feature run: natural (f0,f1)(f2,f3).. or permuted (f0,f4)(f1,f5)(f2,f6)(f3,f7)
          const int at = quarter * 16 + (p.permute_out ? (f & ~7) + 2 * (f & 3) : f & ~1);
          const int r0 = (up ? 1 : 0) + 2 * hi;             // this lane's route of every four
          __nv_bfloat16* dst = orow + (long long)r0 * p.out_stride + at;
          float v[8];
#pragma unroll
          for (int j = 0; j < 16; j += 2) {
            const float mine = __uint_as_float(up ? a[j + 1] : a[j]);
            const float other = __shfl_xor_sync(0xffffffffu, __uint_as_float(up ? a[j] : a[j + 1]), 16);
            v[j >> 1] = up ? silu_f32(other) * mine : silu_f32(mine) * other;
          }
#pragma unroll
          for (int j = 0; j < 8; j += 2) {                  // routes 2j + up and 2j + 2 + up
            const float other = __shfl_xor_sync(0xffffffffu, hi ? v[j] : v[j + 1], swap);
            if (2 * j + r0 < left)
              *reinterpret_cast<uint32_t*>(dst + (long long)(2 * j) * p.out_stride) = hi ? pack_bf16(other, v[j + 1]) : pack_bf16(v[j], other);
          }
        } else if (kSplit && p.k_splits > 1) {
          // float32 sums of this part of the contraction
          float* dst = p.part + t.part * p.part_stride + ((long long)t.row0 + c * 16) * p.n_rows + t.col * kFeatures + quarter * 32 + lane;
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (j < left) dst[(long long)j * p.n_rows] = __uint_as_float(a[j]);
        } else {
          const int hi = lane & 1;
          const float* wr = p.route_weight ? p.route_weight + t.row0 + c * 16 : nullptr;
          const float mine = wr && (lane & 15) < left ? wr[lane & 15] : 1.f;
          __nv_bfloat16* dst = orow + (long long)hi * p.out_stride + quarter * 32 + (lane & ~1);
#pragma unroll
          for (int j = 0; j < 16; j += 2) {
            const float x = __uint_as_float(a[j]) * __shfl_sync(0xffffffffu, mine, j);
            const float y = __uint_as_float(a[j + 1]) * __shfl_sync(0xffffffffu, mine, j + 1);
            const float other = __shfl_xor_sync(0xffffffffu, hi ? x : y, 1);
            if (j + hi < left)
              *reinterpret_cast<uint32_t*>(dst + (long long)j * p.out_stride) = hi ? pack_bf16(other, y) : pack_bf16(x, other);
          }
        }
      }
      tc_fence_before();                                    // every tcgen05.ld of this tile is complete (wait::ld)
      __syncwarp();
      if (lane == 0) mbar_arrive(&sh.acc_empty[buf]);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem, S::kTmemCols);
  }
}

template <int ENC, int MODE, bool WIDE>
int launch_ts(const GroupedGemmArgs& a, GroupedParams p, cudaStream_t stream) {
  using S = TsShape<ENC>;
  auto kernel = grouped_ts_kernel<ENC, MODE, WIDE>;
  constexpr size_t smem = ts_smem_bytes<ENC>();
  static_assert(smem <= 113 * 1024, "two CTAs share an SM");
  static thread_local int configured = -1;
  int dev = 0;
  cudaGetDevice(&dev);
  if (configured != dev) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) { set_error("grouped: cudaFuncSetAttribute: %s", cudaGetErrorString(e)); return ERR_LAUNCH; }
    configured = dev;
  }
  CUtensorMap ma, m0, m1;
  const uint64_t wrows = (uint64_t)a.num_experts * a.n_rows;
  if (ENC == ENC_BF16) {
    const uint32_t box = MODE == 0 ? 16 : kRows;
    if (!make_map(&m0, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, a.w0, (uint64_t)a.k, wrows, kAtomK, box, CU_TENSOR_MAP_SWIZZLE_128B) ||
        !make_map(&m1, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, MODE == 0 ? a.w1 : a.w0, (uint64_t)a.k, wrows, kAtomK, box, CU_TENSOR_MAP_SWIZZLE_128B))
      return ERR_LAUNCH;
  } else {
    const uint64_t rowb = ENC == ENC_Q4 ? a.k / 2 : a.k;
    const uint32_t box = MODE == 0 ? kRows / 2 : kRows;
    const CUtensorMapSwizzle swz = ENC == ENC_Q4 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B;
    if (!make_map(&m0, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, a.w0, rowb, wrows, S::kPackedRow, box, swz) ||
        !make_map(&m1, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, MODE == 0 ? a.w1 : a.w0, rowb, wrows, S::kPackedRow, box, swz))
      return ERR_LAUNCH;
  }
  // with rows fetched by index `act` is [tokens, k] and the map is never used: any valid map will do
  if (!make_map(&ma, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, a.act, (uint64_t)a.k, (uint64_t)(a.gather_route ? kActBox : a.total_rows),
                kAtomK, kActBox, CU_TENSOR_MAP_SWIZZLE_128B))
    return ERR_LAUNCH;
  p.subs = (a.tile_cap + NMAX - 1) / NMAX;
  p.part_major = a.num_experts > 1;
  // An ordinary launch, not a chained one: CTAs that become resident one by one as their predecessor's leave are paired on
  // the SMs by chance, and CTAs with a tile more than the others then meet on one SM (OLMoE Q8, 96 tokens: 127 -> 140 us a
  // layer).  Launched on an empty device, CTA b and b + SMs share an SM and the longer ones spread.
  kernel<<<dim3(2 * sm_count()), S::kThreads, smem, stream>>>(ma, m0, m1, p);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { set_error("grouped: launch failed: %s", cudaGetErrorString(e)); return ERR_LAUNCH; }
  return ERR_NONE;
}

template <int ENC>
int launch_ts(const GroupedGemmArgs& a, const GroupedParams& p, cudaStream_t stream) {
  if (a.tile_cap > NMAX) return a.mode == 0 ? launch_ts<ENC, 0, true>(a, p, stream) : launch_ts<ENC, 1, true>(a, p, stream);
  return a.mode == 0 ? launch_ts<ENC, 0, false>(a, p, stream) : launch_ts<ENC, 1, false>(a, p, stream);
}

}  // namespace

int launch_grouped_gemm_ts(const GroupedGemmArgs& a, cudaStream_t stream) {
  GroupedParams p{};
  p.k = a.k; p.n_rows = a.n_rows;
  p.scales0 = a.s0; p.scales1 = a.s1;
  p.num_tiles = a.num_tiles; p.tile_expert = a.tile_expert; p.tile_row0 = a.tile_row0; p.tile_rows = a.tile_rows;
  p.max_tiles = a.max_tiles;
  p.k_splits = a.k_splits > 1 ? a.k_splits : 1; p.part = a.part; p.part_stride = a.total_rows * a.n_rows;
  p.out = a.out; p.out_stride = a.out_stride; p.route_weight = a.route_weight; p.permute_out = a.permute_out;
  p.status = a.status;
  p.conditional = a.conditional; p.use_ts = a.use_ts;
  if (a.conditional) p.choice = grouped_gemm_choice(a.enc, a.mode == 0 ? a.n_rows : a.k, a.mode == 0 ? a.k : a.n_rows);
  p.gather_route = a.gather_route; p.gather_top_k = a.gather_top_k; p.gather_src = static_cast<const __nv_bfloat16*>(a.act);
  if (a.enc == ENC_Q4) return launch_ts<ENC_Q4>(a, p, stream);
  if (a.enc == ENC_Q8) return launch_ts<ENC_Q8>(a, p, stream);
  if (a.enc == ENC_BF16) return launch_ts<ENC_BF16>(a, p, stream);
  set_error("grouped: unknown encoding %d", a.enc);
  return ERR_BAD_ARGUMENT;
}

}  // namespace umaq
