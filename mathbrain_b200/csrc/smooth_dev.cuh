// Device pieces the smooth forward and backward share.
#pragma once
#include "smooth.cuh"
#include "sm100_ptx.cuh"

namespace mbema {
namespace smooth {

// eight columns of an E row as stored
template <bool EF32> struct ERow { uint4 v[EF32 ? 2 : 1]; };
template <bool EF32>
__device__ __forceinline__ ERow<EF32> load_e(const void* E, size_t off) {
    ERow<EF32> r;
    const uint4* p = reinterpret_cast<const uint4*>(reinterpret_cast<const unsigned char*>(E) + off * (EF32 ? 4 : 2));
#pragma unroll
    for (int i = 0; i < (EF32 ? 2 : 1); ++i) r.v[i] = __ldg(p + i);
    return r;
}
// columns 2p, 2p + 1 as fp16, times 1/4 (see basis())
template <bool EF32>
__device__ __forceinline__ uint32_t e_pair(const ERow<EF32>& r, int p) {
    const uint32_t* u = reinterpret_cast<const uint32_t*>(r.v);
    if (EF32) return ptx::pack_f16x2_sat(__uint_as_float(u[(2 * p) & 7]) * 0.25f, __uint_as_float(u[(2 * p + 1) & 7]) * 0.25f);
    return ptx::pack_f16x2_sat(ptx::bf16_lo(u[p]) * 0.25f, ptx::bf16_hi(u[p]) * 0.25f);
}

// a wait whose outcome is the same for the whole warp (the code after it has warp-wide instructions)
__device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int tag, const unsigned* lim) {
    return __all_sync(0xffffffffu, ptx::mbar_wait(bar, parity, abort_flag, tag, lim));
}

// Gate of eight columns at the four nodes (x: half the pre-activation for SiLU) -> Chebyshev coefficients as fp16 pairs
// and, with DERIV, SiLU' at the nodes as fp16 pairs.
template <bool SILU, bool DERIV>
__device__ __forceinline__ void gate_coefficients(const float (&x)[NJ][8], uint32_t (&cf)[NJ][4], uint32_t (&sp)[DERIV ? NJ : 1][4]) {
    using namespace ptx;
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        f32x2 gt[NJ];
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
            const float h0 = x[j][2 * p], h1 = x[j][2 * p + 1];
            const f32x2 hh = pack2(h0, h1);
            gt[j] = hh;
            if (SILU) {
                const float t0 = tanh_approx(h0), t1 = tanh_approx(h1);
                const f32x2 th = pack2(t0, t1);
                gt[j] = fma2(hh, th, hh);
                if (DERIV) {        // SiLU'(2h) = (1 + t + h (1 - t^2)) / 2
                    const f32x2 u = fma2(pack2(-t0, -t1), th, pack2(1.f, 1.f));
                    const f32x2 d = fma2(fma2(hh, u, th), pack2(0.5f, 0.5f), pack2(0.5f, 0.5f));
                    float lo, hi;
                    unpack2(d, lo, hi);
                    sp[DERIV ? j : 0][p] = pack_f16x2(lo, hi);
                }
            }
        }
        const f32x2 m1 = pack2(-1.f, -1.f), ka = pack2(TAN_PI_8, TAN_PI_8), kn = pack2(-TAN_PI_8, -TAN_PI_8);
        const f32x2 s03 = add2(gt[0], gt[3]), s12 = add2(gt[1], gt[2]);
        const f32x2 d03 = fma2(gt[3], m1, gt[0]), d12 = fma2(gt[2], m1, gt[1]);
        const f32x2 cj[NJ] = {add2(s03, s12), fma2(d12, ka, d03), fma2(s12, m1, s03), fma2(d03, kn, d12)};
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
            float lo, hi;
            unpack2(cj[j], lo, hi);
            cf[j][p] = pack_f16x2_sat(lo, hi);
        }
    }
}

// row t of a 16-column chunk of Q' or dO': v[dd] beta_j scale at column 16 j + dd of a swizzled operand tile
__device__ __forceinline__ void store_basis_rows(unsigned char* tile, int t, const float (&v)[16], const float (&beta)[NJ], float scale) {
    using namespace ptx;
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
        const float s = beta[j] * scale;
#pragma unroll
        for (int g = 0; g < 2; ++g)
            *reinterpret_cast<uint4*>(tile + t * 128 + (((2 * j + g) ^ (t & 7)) << 4)) =
                make_uint4(pack_f16x2_sat(v[8 * g] * s, v[8 * g + 1] * s), pack_f16x2_sat(v[8 * g + 2] * s, v[8 * g + 3] * s),
                           pack_f16x2_sat(v[8 * g + 4] * s, v[8 * g + 5] * s), pack_f16x2_sat(v[8 * g + 6] * s, v[8 * g + 7] * s));
    }
}

}  // namespace smooth
}  // namespace mbema
