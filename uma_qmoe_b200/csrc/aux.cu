// Small supporting kernels: the device-side packer that writes the canonical Q4 / Q8 bytes.
#include "common.cuh"
#include "aux.cuh"

namespace umaq {
namespace {

// Half a warp per 128-element group, lane l of the half owns elements 8l..8l+7; every warp takes kQgLoads pairs of groups
// with all its loads in flight.  blockIdx.y is the chunk of a strided source.
// Bit-identical to the reference's host packer: scale = max|g| / qmax in float32 (1.0 for an
// all-zero group), code = clip(rint(g / scale), -qmax, qmax)
// (src/uma_qmoe/q4.py:136-165, src/uma_qmoe/target_pack.py:92-112 in the reference).
//
// The bound is the stream: 2 bytes read and 0.53 (Q4) or 1.03 (Q8) written per weight; what has to stay below it is the
// number of instructions per weight.  The quotient g / scale is v * inv with inv = 1/scale correctly rounded, corrected once by
// its exact remainder (Markstein, IBM J. Res. Dev. 34, 1990): the correctly rounded quotient, with three operations.  Quotients
// on the boundary between two codes are common, not rare (BF16 weights over a BF16 maximum: one weight in 200), so a path that
// divides next to a boundary is taken by three warps in four.  Groups with a scale below 2^-100 (the remainder would
// underflow), a scale whose mantissa is all ones (excepted by the theorem), an infinity or a NaN divide.
// Measured, 134 M weights to Q4: 87 us (3.9 TB/s); dividing next to a boundary 130, a warp per group with four divisions a
// lane 170.
constexpr int kQgLoads = 4, kQgWarps = 8;
template <int QMAX, bool NIBBLES, bool WIDE>
__global__ void __launch_bounds__(kQgWarps * 32)
quantize_groups_kernel(const __nv_bfloat16* __restrict__ src, long long groups, long long src_stride,
                       uint8_t* __restrict__ codes, float* __restrict__ scales) {
  const int lane = threadIdx.x & 31, l16 = lane & 15;
  const long long first = ((long long)blockIdx.x * kQgWarps + (threadIdx.x >> 5)) * (2 * kQgLoads) + (lane >> 4);
  src += (long long)blockIdx.y * src_stride;
  const long long base = (long long)blockIdx.y * groups;                    // first group of the chunk in the output
  uint4 raw[kQgLoads];
#pragma unroll
  for (int i = 0; i < kQgLoads; ++i) {
    const long long g = first + 2 * i;
    raw[i] = make_uint4(0, 0, 0, 0);
    if (g < groups) {
      const __nv_bfloat16* at = src + g * 128 + l16 * 8;
      if (WIDE) {
        raw[i] = __ldcs(reinterpret_cast<const uint4*>(at));                // read once: not worth keeping in L2
      } else {
        const uint2 lo = reinterpret_cast<const uint2*>(at)[0], hi = reinterpret_cast<const uint2*>(at)[1];
        raw[i] = make_uint4(lo.x, lo.y, hi.x, hi.y);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < kQgLoads; ++i) {
    const long long g = first + 2 * i;
    const uint32_t w[4] = {raw[i].x, raw[i].y, raw[i].z, raw[i].w};
    // |g| of two BF16 values at a time: their bits without the signs order like the values (a NaN above everything)
    uint32_t m2 = __vmaxu2(__vmaxu2(w[0] & 0x7fff7fffu, w[1] & 0x7fff7fffu), __vmaxu2(w[2] & 0x7fff7fffu, w[3] & 0x7fff7fffu));
#pragma unroll
    for (int o = 8; o; o >>= 1) m2 = __vmaxu2(m2, __shfl_xor_sync(0xffffffffu, m2, o));
    const uint32_t m1 = max(m2 << 16, m2 & 0xffff0000u);
    float am = __uint_as_float(m1);
    bool divide = m1 > 0x7f800000u;
    if (__any_sync(0xffffffffu, divide)) {                                  // a NaN somewhere: fmaxf passes over it
      am = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j)
        am = fmaxf(am, fmaxf(fabsf(__uint_as_float(w[j] << 16)), fabsf(__uint_as_float(w[j] & 0xffff0000u))));
#pragma unroll
      for (int o = 8; o; o >>= 1) am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, o));
    }
    float scale = __fdiv_rn(am, (float)QMAX);
    if (scale == 0.f) scale = 1.f;
    const float inv = __frcp_rn(scale);
    constexpr float kMagic = 12582912.f;                                    // 1.5 * 2^23: the ulp of a sum with it is 1
    divide = divide || !(scale > 7.8886091e-31f) || !(am < 3.0e38f) || (__float_as_uint(scale) & 0x7fffffu) == 0x7fffffu;
    float n[8];                                                             // minus the code
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float v = __uint_as_float(j & 1 ? w[j >> 1] & 0xffff0000u : w[j >> 1] << 16);
      const float q0 = __fmul_rn(v, inv);
      const float q = __fmaf_rn(__fmaf_rn(-q0, scale, v), inv, q0);
      n[j] = kMagic - __fadd_rn(q, kMagic);                                 // nearest integer, ties to even
    }
    if (divide) {
#pragma unroll 1
      for (int j = 0; j < 8; ++j) {
        const uint32_t word = j < 4 ? (j < 2 ? w[0] : w[1]) : (j < 6 ? w[2] : w[3]);
        float r = rintf(__fdiv_rn(__uint_as_float(j & 1 ? word & 0xffff0000u : word << 16), scale));
        r = -fminf(fmaxf(r, (float)-QMAX), (float)QMAX);
#pragma unroll
        for (int k = 0; k < 8; ++k)
          if (k == j) n[k] = r;
      }
    }
    if (g >= groups) continue;
    if (NIBBLES) {
      // four codes as one float sum of code * 16^j, exact below 2^16; + 8 in every nibble, then ^ 8 = two's complement
      const float lo = -fmaf(fmaf(fmaf(n[3], 16.f, n[2]), 16.f, n[1]), 16.f, n[0]);
      const float hi = -fmaf(fmaf(fmaf(n[7], 16.f, n[6]), 16.f, n[5]), 16.f, n[4]);
      const uint32_t o = prmt(__float_as_uint(lo + (kMagic + 0x8888)), __float_as_uint(hi + (kMagic + 0x8888)), 0x5410) ^ 0x88888888u;
      uint8_t* dst = codes + (base + g) * 64 + l16 * 4;
      if (WIDE) {
        *reinterpret_cast<uint32_t*>(dst) = o;
      } else {
        reinterpret_cast<uint16_t*>(dst)[0] = (uint16_t)o;
        reinterpret_cast<uint16_t*>(dst)[1] = (uint16_t)(o >> 16);
      }
    } else {
      uint32_t q[8];                                                        // two's complement in the low byte
#pragma unroll
      for (int j = 0; j < 8; ++j) q[j] = __float_as_uint(kMagic - n[j]);
      const uint32_t lo = prmt(prmt(q[0], q[1], 0x0040), prmt(q[2], q[3], 0x0040), 0x5410);
      const uint32_t hi = prmt(prmt(q[4], q[5], 0x0040), prmt(q[6], q[7], 0x0040), 0x5410);
      uint8_t* dst = codes + (base + g) * 128 + l16 * 8;
      if (WIDE) {
        *reinterpret_cast<uint2*>(dst) = make_uint2(lo, hi);
      } else {
        reinterpret_cast<uint32_t*>(dst)[0] = lo;
        reinterpret_cast<uint32_t*>(dst)[1] = hi;
      }
    }
    if (l16 == 0) scales[base + g] = scale;
  }
}

template <int QMAX, bool NIBBLES>
void run_quantize(const __nv_bfloat16* src, long long groups, long long chunks, long long src_stride, uint8_t* codes,
                  float* scales, cudaStream_t stream) {
  const long long per_block = kQgWarps * 2 * kQgLoads;
  const dim3 grid((unsigned)((groups + per_block - 1) / per_block), (unsigned)chunks);
  // 16-byte loads and one store per lane where the pointers allow it; otherwise the 8-byte loads and the smaller stores
  // that any tensor of the types in question can take
  const bool wide = !(reinterpret_cast<uintptr_t>(src) & 15) && !(src_stride & 7) &&
                    !(reinterpret_cast<uintptr_t>(codes) & (NIBBLES ? 3 : 7));
  if (wide) quantize_groups_kernel<QMAX, NIBBLES, true><<<grid, kQgWarps * 32, 0, stream>>>(src, groups, src_stride, codes, scales);
  else quantize_groups_kernel<QMAX, NIBBLES, false><<<grid, kQgWarps * 32, 0, stream>>>(src, groups, src_stride, codes, scales);
}

}  // namespace

int launch_quantize_groups(const void* src_bf16, long long chunk_elements, long long chunks, long long chunk_stride, int enc,
                           void* codes, float* scales, cudaStream_t stream) {
  if (!src_bf16 || !codes || !scales || chunk_elements <= 0 || chunk_elements % 128) {
    set_error("quantize: element count must be a positive multiple of 128");
    return ERR_BAD_ARGUMENT;
  }
  if ((reinterpret_cast<uintptr_t>(src_bf16) & 7) || (chunk_stride & 3) || (reinterpret_cast<uintptr_t>(scales) & 3) ||
      (reinterpret_cast<uintptr_t>(codes) & (enc == ENC_Q4 ? 1 : 3))) {
    set_error("quantize: misaligned pointer or chunk stride");
    return ERR_BAD_ARGUMENT;
  }
  if (chunks < 1 || chunks > 65535 || chunk_stride < 0) { set_error("quantize: between 1 and 65535 chunks"); return ERR_BAD_ARGUMENT; }
  const long long groups = chunk_elements / 128;
  if ((groups + 7) / 8 > 0x7fffffffLL) { set_error("quantize: tensor too large"); return ERR_BAD_ARGUMENT; }
  const __nv_bfloat16* s = static_cast<const __nv_bfloat16*>(src_bf16);
  if (enc == ENC_Q4) run_quantize<7, true>(s, groups, chunks, chunk_stride, static_cast<uint8_t*>(codes), scales, stream);
  else if (enc == ENC_Q8) run_quantize<127, false>(s, groups, chunks, chunk_stride, static_cast<uint8_t*>(codes), scales, stream);
  else { set_error("quantize: encoding must be Q4 or Q8"); return ERR_BAD_ARGUMENT; }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { set_error("quantize: launch failed: %s", cudaGetErrorString(e)); return ERR_LAUNCH; }
  return ERR_NONE;
}

}  // namespace umaq
