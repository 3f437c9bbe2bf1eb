// Flash-EMA attention forward over smooth slot states (see smooth.cuh): one CTA per (tile, head, sample).
//
// Items are walked in blocks of 128, a head's 64 columns in chunks of 16 (16 columns x 4 coefficients = one 64-wide
// swizzle atom).  Per block, on the tensor cores:
//     pre_c [128 items x 64]  = A . W'_c            A: item states, W'_c: W_pe scaled to the four nodes
//     S     [128 steps x 128] += Q'_c . K_c^T       K_c = E_k c_j, written by the gate warps
//     O'_c  [128 steps x 64]  += P . V_c            P from tensor memory, V_c = E_v c_j
// Warps: two gate warpgroups (a thread per item; half of a chunk's columns each), two softmax warpgroups (a thread per
// step and half a block's items), one loader (bulk copies of A and W' images), and a lane each for the gate products, S
// and P.V, so that none waits for another's operands.  All hand-offs are mbarriers with bounded waits.
//
// The gate warps are the longest stage (some 1450 cycles a chunk, 5800 a block: 4 * 64 tanh an item and their coefficients), so
// everything else is laid out to run beside them: scores and P have tensor memory of their own (the next block's S starts while P.V
// reads P; the gate product has one accumulator, read at once), and V has six chunks (five for 128 channels, where the states take
// the room) of which the gate runs two ahead of P.V.  With P over S and four V chunks a block took S, softmax, P.V and gate one
// after the other: 1.05 ms a layer at B=56, T=512, N=64, 0.86 ms so; 1.14 and 1.03 ms at B=8, T=4096, N=128.
#include "smooth.cuh"
#include "smooth_dev.cuh"

namespace mbema {
namespace smooth {

using namespace ptx;

namespace fwd {

static constexpr int GATE_WARPS = 8, SM_WARPS = 8;
static constexpr int W_LOAD = 16, W_GATE = 17, W_SCORE = 18, W_PV = 19;
static constexpr int THREADS = 20 * 32;      // launched with 96 registers a thread: 61440 = 4 * 128 * 104 + 128 * 64
static constexpr uint32_t T_O = 0, T_S = 256, T_P = 384, T_PRE = 448;     // tensor-memory columns
static constexpr float RESCALE = 8.0f;      // log2 units the softmax reference may lag behind (P <= 2^8 in fp16)

struct Bars {
    uint64_t a_full, a_free, w_full[2], w_free[2], pre_full, pre_empty, kv_full[NCH], k_free[2], v_free[6];
    uint64_t s_full, s_free, p_full, mx_full, v_full, pv_done, o_full, drain;
    uint32_t tmem_base;
    int abort_flag, drain_flag;
    unsigned spin_limit;
};

template <int NK> struct L {
    static constexpr int NV = NK == 1 ? 6 : 5;          // V chunks in flight
    static constexpr int Q = 0, A = Q + NCH * ATOM, W = A + NK * ATOM, K = W + 2 * WPIECE, V = K + 2 * ATOM, MX = V + NV * ATOM,
                         BAR = MX + 4 * TM * 4, SMEM = BAR + 512;
    static_assert(sizeof(Bars) <= 512 && SMEM <= 227 * 1024, "shared memory");
};

template <bool SILU, int NK, bool EF32>
__global__ void __launch_bounds__(THREADS, 1) k_smooth_fwd(FlashArgs a, Items it, Ws w, int* status) {
    extern __shared__ __align__(1024) unsigned char sm[];
    using M = L<NK>;
    Bars* bars = reinterpret_cast<Bars*>(sm + M::BAR);
    float* mx_sh = reinterpret_cast<float*>(sm + M::MX);
    volatile int* abort_flag = &bars->abort_flag;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tile = blockIdx.x, h = blockIdx.y, b = a.order ? a.order[blockIdx.z] : (int)blockIdx.z;
    const int bt = b * a.nT + tile, t0 = tile * TM, D = a.H * HD;
    const int Lb = a.seq_lens ? min(max(a.seq_lens[b], 0), a.T) : a.T;
    const int level = w.level[bt];
    if (level == LEVEL_EXACT) return;
    if (smem_u32(sm) & 1023u) {        // the swizzled tiles need it; there is no room to align by hand
        if (tid == 0) atomicOr(status, 1 | (31 << 8));
        return;
    }
    const size_t row0 = ((size_t)b * a.H + h) * a.T + t0;
    if (t0 >= Lb) {          // a tile beyond the valid length
        for (int i = tid; i < min(TM, a.T - t0) * (HD / 4); i += THREADS)
            *reinterpret_cast<float4*>(a.O + (row0 + i / (HD / 4)) * HD + (i % (HD / 4)) * 4) = make_float4(0.f, 0.f, 0.f, 0.f);
        if (tid < min(TM, a.T - t0)) a.LSE[row0 + tid] = 0.f;
        return;
    }
    if (tid == 0) {
        mbar_init(&bars->a_full, 1); mbar_init(&bars->a_free, 1);
        mbar_init(&bars->pre_full, 1); mbar_init(&bars->pre_empty, GATE_WARPS);
        for (int i = 0; i < 2; ++i) { mbar_init(&bars->w_full[i], 1); mbar_init(&bars->w_free[i], 1); mbar_init(&bars->k_free[i], 1); }
        for (int i = 0; i < NCH; ++i) mbar_init(&bars->kv_full[i], GATE_WARPS);
        for (int i = 0; i < M::NV; ++i) mbar_init(&bars->v_free[i], 1);
        mbar_init(&bars->s_full, 1); mbar_init(&bars->s_free, SM_WARPS); mbar_init(&bars->p_full, SM_WARPS);
        mbar_init(&bars->mx_full, SM_WARPS); mbar_init(&bars->v_full, 1); mbar_init(&bars->pv_done, 1);
        mbar_init(&bars->o_full, 1); mbar_init(&bars->drain, 3);
        bars->abort_flag = *reinterpret_cast<volatile int*>(status);      // an earlier CTA gave up: do nothing
        bars->drain_flag = 0;
        bars->spin_limit = a.test_withhold ? 64u : MBEMA_SPIN_LIMIT;
        fence_barrier_init();
    }
    if (warp == W_GATE) {
        tmem_alloc(&bars->tmem_base, 512);
        tmem_relinquish();
    }
    // Q' tiles: row t, chunk c holds q[16 c + dd] beta_j(t) log2(e) / 8 at column 16 j + dd
    if (tid < TM * NCH) {
        const int t = tid & (TM - 1), c = tid >> 7;
        float beta[NJ], q[16];
        basis(t, level, beta);
#pragma unroll
        for (int i = 0; i < 16; i += 4) {
            const float4 v = t0 + t < Lb ? ld4_dyn_f32(a.Q, a.q_dt, (row0 + t) * HD + c * 16 + i) : make_float4(0.f, 0.f, 0.f, 0.f);
            q[i] = v.x; q[i + 1] = v.y; q[i + 2] = v.z; q[i + 3] = v.w;
        }
        store_basis_rows(sm + M::Q + c * ATOM, t, q, beta, 0.125f * 1.4426950409f);
    }
    fence_proxy_async_smem();
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = bars->tmem_base;
    const int n_blk = a.hot ? it.count[bt].y : it.count[bt].w;        // the hot slots' blocks are the last ones
    const int n_it = bars->abort_flag ? 0 : n_blk << level;        // blocks of segment 0, then of segment 1, ...
    const unsigned* lim = &bars->spin_limit;

    if (warp < GATE_WARPS) {
        // ======================================================== gate: item r, columns 8 wg .. 8 wg + 7 of every chunk
        asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");
        const int wg = warp >> 2, r = tid & 127;
        const uint32_t t_pre = tmem + ((uint32_t)((warp & 3) * 32) << 16) + T_PRE + wg * 8;
        const int2* meta = it.meta + (size_t)bt * it.IB * IBLK + r;
        const int x7 = r & 7;
        size_t eo = 0;          // this item's E columns of chunk 0
        ERow<EF32> ek, ev;
        if (n_it > 0) {
            eo = e_row(a, b, __ldg(&meta[0].x)) * D + h * HD + wg * 8;
            ek = load_e<EF32>(a.Ek, eo);
            ev = load_e<EF32>(a.Ev, eo);
        }
        bool alive = true;
        for (int i = 0; i < n_it && alive; ++i) {
#pragma unroll 1
            for (int c = 0; c < NCH; ++c) {
                // the next chunk's E columns fly while this chunk is worked on
                ERow<EF32> nk = ek, nv = ev;
                if (c == NCH - 1 && i + 1 < n_it) eo = e_row(a, b, __ldg(&meta[(size_t)((i + 1) % n_blk) * IBLK].x)) * D + h * HD + wg * 8;
                if (c < NCH - 1 || i + 1 < n_it) {
                    const size_t off = eo + ((c + 1) & (NCH - 1)) * 16;
                    nk = load_e<EF32>(a.Ek, off);
                    nv = load_e<EF32>(a.Ev, off);
                }
                const int st = c & 1, use = 2 * i + (c >> 1), n = 4 * i + c;
                if (!(alive = warp_wait(&bars->pre_full, (uint32_t)(n & 1), abort_flag, 1, lim))) break;
                tc_fence_after_sync();
                float x[NJ][8];
#pragma unroll
                for (int j = 0; j < NJ; ++j) tmem_ld_32x32b_x8(t_pre + j * 16, x[j]);
                tmem_wait_ld();
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0 && !(a.test_withhold && n == 0)) mbar_arrive(&bars->pre_empty);
                uint32_t cf[NJ][4], none[1][4];
                gate_coefficients<SILU, false>(x, cf, none);
                if (use >= 1 && !(alive = warp_wait(&bars->k_free[st], (uint32_t)((use - 1) & 1), abort_flag, 2, lim))) break;
                unsigned char* kd = sm + M::K + st * ATOM + r * 128;
                uint32_t e2[4], f2[4];
#pragma unroll
                for (int p = 0; p < 4; ++p) { e2[p] = e_pair<EF32>(ek, p); f2[p] = e_pair<EF32>(ev, p); }
#pragma unroll
                for (int j = 0; j < NJ; ++j)
                    st_shared_v4(kd + (((2 * j + wg) ^ x7) << 4), mul_f16x2(cf[j][0], e2[0]), mul_f16x2(cf[j][1], e2[1]), mul_f16x2(cf[j][2], e2[2]), mul_f16x2(cf[j][3], e2[3]));
                const int vb = n % M::NV;
                if (n >= M::NV && !(alive = warp_wait(&bars->v_free[vb], (uint32_t)((n / M::NV - 1) & 1), abort_flag, 3, lim))) break;
                unsigned char* vd = sm + M::V + vb * ATOM + r * 128;
#pragma unroll
                for (int j = 0; j < NJ; ++j)
                    st_shared_v4(vd + (((2 * j + wg) ^ x7) << 4), mul_f16x2(cf[j][0], f2[0]), mul_f16x2(cf[j][1], f2[1]), mul_f16x2(cf[j][2], f2[2]), mul_f16x2(cf[j][3], f2[3]));
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(&bars->kv_full[c]);
                ek = nk;
                ev = nv;
            }
        }
    } else if (warp < GATE_WARPS + SM_WARPS) {
        // ======================================================== softmax: step `row`, items 64 half .. 64 half + 63
        asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");
        const int half = (warp >> 2) & 1, row = tid & 127;
        const uint32_t t_row = tmem + ((uint32_t)((warp & 3) * 32) << 16);
        const float rest = a.v_total - (float)a.kcount[b];
        float m, l = 0.f;
        if (!a.listed_only && rest > 0.f) { m = 0.f; l = half == 0 ? rest : 0.f; } else m = -INFINITY;
        const uint2* mask = reinterpret_cast<const uint2*>(it.mask + (size_t)bt * it.IB * IBLK + row) + half;
        const int my_seg = row / (TM >> level);
        uint2 mk = n_it > 0 ? __ldg(mask) : make_uint2(0u, 0u);
        bool alive = true;
        for (int i = 0; i < n_it; ++i) {
            uint2 mcur = mk;
            if (i / n_blk != my_seg) mcur = make_uint2(0u, 0u);
            if (i + 1 < n_it) mk = __ldg(mask + (size_t)((i + 1) % n_blk) * IBLK * 2);
            if (!(alive = warp_wait(&bars->s_full, (uint32_t)(i & 1), abort_flag, 4, lim))) break;
            tc_fence_after_sync();
            float s[64];
            tmem_ld_32x32b_x32(t_row + T_S + half * 64, s);
            tmem_ld_32x32b_x32(t_row + T_S + half * 64 + 32, s + 32);
            tmem_wait_ld();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars->s_free);          // the next block's scores may be written
            if (!__all_sync(0xffffffffu, (mcur.x & mcur.y) == 0xffffffffu)) {
#pragma unroll
                for (int k = 0; k < 32; ++k) {
                    s[k] = (mcur.x >> k) & 1u ? s[k] : -INFINITY;
                    s[k + 32] = (mcur.y >> k) & 1u ? s[k + 32] : -INFINITY;
                }
            }
            float b0 = -INFINITY, b1 = -INFINITY;
#pragma unroll
            for (int k = 0; k < 64; k += 4) {
                b0 = fmaxf(b0, fmaxf(s[k], s[k + 1]));
                b1 = fmaxf(b1, fmaxf(s[k + 2], s[k + 3]));
            }
            float* mx = mx_sh + (i & 1) * 2 * TM;
            mx[half * TM + row] = fmaxf(b0, b1);
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars->mx_full);
            if (!(alive = warp_wait(&bars->mx_full, (uint32_t)(i & 1), abort_flag, 5, lim))) break;
            // the products of the block before have read P and left O'
            if (i >= 1 && !(alive = warp_wait(&bars->pv_done, (uint32_t)((i - 1) & 1), abort_flag, 17, lim))) break;
            tc_fence_after_sync();
            const float mb = fmaxf(fmaxf(b0, b1), mx[(half ^ 1) * TM + row]);
            const bool up = mb > m + RESCALE;
            if (__any_sync(0xffffffffu, up)) {
                const float al = up ? ex2_approx(m - mb) : 1.0f;       // m = -inf: 0
                l *= al;
                if (up) m = mb;
                if (i > 0) {       // this half's columns of O'
#pragma unroll 1
                    for (int k = 0; k < 128; k += 16) {
                        float o[16];
                        tmem_ld_32x32b_x16(t_row + T_O + half * 128 + k, o);
                        tmem_wait_ld();
#pragma unroll
                        for (int e = 0; e < 16; ++e) o[e] *= al;
                        tmem_st_32x32b_x16(t_row + T_O + half * 128 + k, o);
                    }
                }
            }
            const float mm = m == -INFINITY ? 0.f : m;
            float l0 = 0.f, l1 = 0.f;
            // P as fp16 pairs
#pragma unroll
            for (int k = 0; k < 64; k += 16) {
                uint32_t p2[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const float p = ex2_approx(s[k + 2 * e] - mm), q = ex2_approx(s[k + 2 * e + 1] - mm);
                    l0 += p; l1 += q;
                    p2[e] = pack_f16x2(p, q);
                }
                tmem_st_x8(t_row + T_P + half * 32 + k / 2, p2);
            }
            l += l0 + l1;
            tmem_wait_st();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars->p_full);
        }
        if (alive && n_it > 0) alive = warp_wait(&bars->o_full, 0u, abort_flag, 6, lim);
        if (alive && __all_sync(0xffffffffu, !*abort_flag)) {
            tc_fence_after_sync();
            float* mx = mx_sh + (n_it & 1) * 2 * TM;
            mx[half * TM + row] = l;
            // the hot slots' share, from the every-step kernel
            const bool merge = a.hot && a.hot[bt * (HOT + 1)] > 0 && t0 + row < Lb;
            const float mh = merge ? a.LSE[row0 + row] * 1.4426950409f : -INFINITY;
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars->mx_full);
            alive = warp_wait(&bars->mx_full, (uint32_t)(n_it & 1), abort_flag, 7, lim);
            l += mx[(half ^ 1) * TM + row];
            const float mm = fmaxf(m, mh), wc = m == -INFINITY ? 0.f : exp2f(m - mm), wh = merge ? exp2f(mh - mm) : 0.f;
            l = fmaf(l, wc, wh);
            const bool ok = t0 + row < Lb && l > 0.f;
            const float inv = ok ? wc / l : 0.f, inv_h = ok ? wh / l : 0.f;
            float beta[NJ];
            basis(row, level, beta);
#pragma unroll 1
            for (int c = half * 2; c < half * 2 + 2; ++c) {
                float o[64];
                if (n_it > 0) {
                    tmem_ld_32x32b_x32(t_row + T_O + c * 64, o);
                    tmem_ld_32x32b_x32(t_row + T_O + c * 64 + 32, o + 32);
                    tmem_wait_ld();
                } else {
#pragma unroll
                    for (int e = 0; e < 64; ++e) o[e] = 0.f;
                }
                if (alive && t0 + row < a.T) {
#pragma unroll
                    for (int d = 0; d < 16; d += 4) {
                        float v[4];
                        float4* out = reinterpret_cast<float4*>(a.O + (row0 + row) * HD + c * 16 + d);
                        const float4 oh = merge ? *out : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const int k = d + e;
                            v[e] = ok ? inv * fmaf(beta[3], o[48 + k], fmaf(beta[2], o[32 + k], fmaf(beta[1], o[16 + k], o[k]))) : 0.f;
                        }
                        *out = make_float4(fmaf(inv_h, oh.x, v[0]), fmaf(inv_h, oh.y, v[1]), fmaf(inv_h, oh.z, v[2]), fmaf(inv_h, oh.w, v[3]));
                    }
                }
            }
            if (alive && half == 0 && t0 + row < a.T) a.LSE[row0 + row] = ok ? mm * 0.6931471806f + logf(l) : 0.f;
        }
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
        if (warp == W_LOAD && lane == 0) {
            // ==================================================== loader
            const unsigned char* img = it.a_img + (size_t)bt * it.IB * NK * ATOM;
            int np = 0, na = 0;
            bool alive = true;
            for (int i = 0; i < n_it && alive; ++i) {
                const int seg = i / n_blk, blk = i - seg * n_blk;
                const unsigned char* wi = w.w_img + (size_t)((((1 << level) - 1 + seg) * a.H + h) * NCH) * NK * WPIECE;
                if (i >= 1 && !(alive = mbar_wait(&bars->a_free, (uint32_t)((i - 1) & 1), abort_flag, 8, lim))) break;
                mbar_expect_tx(&bars->a_full, NK * ATOM);
                bulk_load(sm + M::A, img + (size_t)blk * NK * ATOM, NK * ATOM, &bars->a_full);
                ++na;
                for (int p = 0; p < NCH * NK; ++p, ++np) {
                    const int sw = np & 1, uw = np >> 1;
                    if (uw >= 1 && !(alive = mbar_wait(&bars->w_free[sw], (uint32_t)((uw - 1) & 1), abort_flag, 9, lim))) break;
                    mbar_expect_tx(&bars->w_full[sw], WPIECE);
                    bulk_load(sm + M::W + sw * WPIECE, wi + (size_t)p * WPIECE, WPIECE, &bars->w_full[sw]);
                }
            }
            // no copy of this CTA is in flight when it ends
            if (na > 0) mbar_wait<100>(&bars->a_full, (uint32_t)((na - 1) & 1), &bars->drain_flag, 10);
            for (int s = 0; s < 2; ++s)
                if (np > s) mbar_wait<100>(&bars->w_full[s], (uint32_t)(((np - 1 - s) >> 1) & 1), &bars->drain_flag, 10);
        } else if (warp == W_GATE && lane == 0) {
            // ==================================================== gate products
            const uint32_t idesc = umma_idesc_16(IBLK, 64, 0, 0, 0, 0);
            int np = 0;
            bool alive = true;
            for (int i = 0; i < n_it && alive; ++i) {
                if (!(alive = mbar_wait(&bars->a_full, (uint32_t)(i & 1), abort_flag, 11, lim))) break;
                for (int c = 0; c < NCH && alive; ++c) {
                    const int n = 4 * i + c;
                    if (n >= 1 && !(alive = mbar_wait(&bars->pre_empty, (uint32_t)((n - 1) & 1), abort_flag, 12, lim))) break;
                    for (int p = 0; p < NK; ++p, ++np) {
                        if (!(alive = mbar_wait(&bars->w_full[np & 1], (uint32_t)((np >> 1) & 1), abort_flag, 13, lim))) break;
                        tc_fence_after_sync();
                        const uint32_t ab = smem_u32(sm + M::A + p * ATOM), wb = smem_u32(sm + M::W + (np & 1) * WPIECE);
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            umma_bf16_ss(tmem + T_PRE, umma_desc_k_sw128(ab + k * 32), umma_desc_k_sw128(wb + k * 32), idesc, (p | k) != 0);
                        umma_commit(&bars->w_free[np & 1]);
                    }
                    if (alive) umma_commit(&bars->pre_full);
                }
                if (alive) umma_commit(&bars->a_free);
            }
            umma_commit(&bars->drain);
        } else if (warp == W_SCORE && lane == 0) {
            // ==================================================== S
            const uint32_t id_s = umma_idesc_16(TM, IBLK, 0, 0, 0, 0);
            const uint32_t qb = smem_u32(sm + M::Q), kb = smem_u32(sm + M::K);
            bool alive = true;
            for (int i = 0; i < n_it && alive; ++i) {
                if (i >= 1 && !(alive = mbar_wait(&bars->s_free, (uint32_t)((i - 1) & 1), abort_flag, 18, lim))) break;
                for (int c = 0; c < NCH; ++c) {
                    if (!(alive = mbar_wait(&bars->kv_full[c], (uint32_t)(i & 1), abort_flag, 14, lim))) break;
                    tc_fence_after_sync();
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        umma_bf16_ss(tmem + T_S, umma_desc_k_sw128(qb + c * ATOM + k * 32), umma_desc_k_sw128(kb + (c & 1) * ATOM + k * 32), id_s, (c | k) != 0);
                    umma_commit(&bars->k_free[c & 1]);
                }
                if (!alive) break;
                mbar_arrive(&bars->v_full);          // the block's V chunks, seen here on kv_full, for the lane that reads them
                umma_commit(&bars->s_full);
            }
            umma_commit(&bars->drain);
        } else if (warp == W_PV && lane == 0) {
            // ==================================================== P.V
            const uint32_t id_o = umma_idesc_16(TM, 64, 0, 1, 0, 0), vb = smem_u32(sm + M::V);
            bool alive = true;
            for (int i = 0; i < n_it && alive; ++i) {
                if (!(alive = mbar_wait(&bars->v_full, (uint32_t)(i & 1), abort_flag, 19, lim))) break;
                if (!(alive = mbar_wait(&bars->p_full, (uint32_t)(i & 1), abort_flag, 15, lim))) break;
                tc_fence_after_sync();
                for (int c = 0; c < NCH; ++c) {
                    const int slot = (4 * i + c) % M::NV;
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                        umma_16_ts(tmem + T_O + c * 64, tmem + T_P + k * 8, umma_desc_mn_sw128(vb + slot * ATOM + k * 2048, ATOM, 1024), id_o, (i | k) != 0);
                    umma_commit(&bars->v_free[slot]);
                }
                umma_commit(&bars->pv_done);
            }
            umma_commit(&bars->o_full);
            umma_commit(&bars->drain);
        }
    }
    // ---------------------------------------------------------------- teardown
    tc_fence_before_sync();
    __syncthreads();
    if (warp == W_GATE) {
        mbar_wait<100>(&bars->drain, 0u, &bars->drain_flag, 16);
        tc_fence_after_sync();
        tmem_dealloc(tmem, 512);
    }
    if (tid == 0 && (bars->abort_flag | bars->drain_flag)) atomicOr(status, bars->abort_flag | bars->drain_flag);
}

}  // namespace fwd

int forward(const FlashArgs& a, const Items& it, const Ws& w, int* status, cudaStream_t st) {
    const dim3 grid(a.nT, a.H, a.B);
#define MBEMA_SMOOTH(S_, NK_, E_)                                                                                             \
    do {                                                                                                                       \
        MBEMA_CUDA_TRY(cudaFuncSetAttribute(fwd::k_smooth_fwd<S_, NK_, E_>, cudaFuncAttributeMaxDynamicSharedMemorySize, fwd::L<NK_>::SMEM)); \
        fwd::k_smooth_fwd<S_, NK_, E_><<<grid, fwd::THREADS, fwd::L<NK_>::SMEM, st>>>(a, it, w, status);                                    \
    } while (0)
#define MBEMA_SMOOTH_E(S_, NK_) do { if (a.e_dt == MBEMA_F32) MBEMA_SMOOTH(S_, NK_, true); else MBEMA_SMOOTH(S_, NK_, false); } while (0)
    if (a.N == 64) { if (a.silu) MBEMA_SMOOTH_E(true, 1); else MBEMA_SMOOTH_E(false, 1); }
    else { if (a.silu) MBEMA_SMOOTH_E(true, 2); else MBEMA_SMOOTH_E(false, 2); }
#undef MBEMA_SMOOTH_E
#undef MBEMA_SMOOTH
    return check_launch();
}

}  // namespace smooth
}  // namespace mbema
