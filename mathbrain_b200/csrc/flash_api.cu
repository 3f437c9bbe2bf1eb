// C entry points of the flash-EMA attention: argument checks and dispatch on the compute mode.
#include "flash.cuh"
#include "smooth.cuh"

using namespace mbema;

static bool dt_ok(int dt) { return dt == MBEMA_F32 || dt == MBEMA_BF16; }

static int flash_check(int64_t B, int64_t H, int64_t T, int64_t hd, int64_t N, int64_t K, int mode) {
    if (B < 0 || H < 1 || T < 1 || N < 1 || K < 1) return MBEMA_ERR_SHAPE;
    if (hd != 64 || N > 128 || T > 8192 || B > 65535 || H > 65535) return MBEMA_ERR_UNSUPPORTED;
    if (mode != MBEMA_MODE_FP32 && mode != MBEMA_MODE_TC_BF16) return MBEMA_ERR_UNSUPPORTED;
    if (mode == MBEMA_MODE_TC_BF16 && !flash_tc_supported((int)H, (int)N, (int)K)) return MBEMA_ERR_UNSUPPORTED;
    return MBEMA_OK;
}

static FlashArgs pack(const void* Q, int q_dtype, const int64_t* x, const void* E_k, const void* E_v, int e_dtype,
                      const float* W_pe, const float* rhos, const int64_t* unique, const float* tile_state,
                      const float* tok_state, const int32_t* kcount, const int32_t* seq_lens, int64_t B, int64_t H,
                      int64_t T, int64_t N, int64_t K, int64_t V_total, int flags) {
    FlashArgs a{};
    a.Q = Q; a.q_dt = q_dtype; a.x = (const long long*)x; a.Ek = E_k; a.Ev = E_v; a.e_dt = e_dtype;
    a.W = W_pe; a.rhos = rhos; a.unique = (const long long*)unique; a.tile_state = tile_state;
    a.tok_state = tok_state; a.kcount = kcount; a.seq_lens = seq_lens;
    a.order = kcount ? kcount + B : nullptr;
    a.B = (int)B; a.H = (int)H; a.T = (int)T; a.N = (int)N; a.K = (int)K;
    a.nT = (int)((T + MBEMA_TILE_T - 1) / MBEMA_TILE_T);
    a.v_total = (float)V_total;
    a.silu = (flags & MBEMA_FLAG_SILU) ? 1 : 0;
    a.listed_only = (flags & MBEMA_FLAG_LISTED_ONLY) ? 1 : 0;
    a.test_withhold = (flags & MBEMA_FLAG_TEST_WITHHOLD_ARRIVE) ? 1 : 0;
    a.erow = nullptr;
    a.e_rows = (long long)B * K;
    return a;
}

// offset of the items block of mbema_tile_items behind the snapshots
static size_t items_offset(int64_t B, int64_t T, int64_t N, int64_t K) {
    return align_up((size_t)B * ((T + MBEMA_TILE_T - 1) / MBEMA_TILE_T) * K * N * 6, 1024);
}

extern "C" size_t mbema_tile_items_bytes(int64_t B, int64_t T, int64_t N, int64_t K) {
    return (N == 64 || N == 128) && flash_tc_supported(2, (int)N, (int)K) ? items_offset(B, T, N, K) + smooth::items_bytes(B, T, N, K) : 0;
}

extern "C" int mbema_tile_items(const int64_t* x, const int64_t* unique, const float* rhos, float* tile_state, const float* tok_state,
                                const int32_t* kcount, const int32_t* seq_lens, int64_t B, int64_t T, int64_t N, int64_t K,
                                void* stream) {
    if (B < 0 || T < 1 || N < 1 || K < 1) return MBEMA_ERR_SHAPE;
    if (T > 8192 || B > 65535 || mbema_tile_items_bytes(B, T, N, K) == 0) return MBEMA_ERR_UNSUPPORTED;
    if (B == 0) return MBEMA_OK;
    if (!x || !unique || !rhos || !tile_state || !tok_state || !kcount) return MBEMA_ERR_NULL;
    if (((uintptr_t)tile_state & 1023) || ((uintptr_t)tok_state & 15)) return MBEMA_ERR_ALIGN;
    const FlashArgs a = pack(nullptr, 0, x, nullptr, nullptr, 0, nullptr, rhos, unique, tile_state, tok_state, kcount, seq_lens, B, 1, T,
                             N, K, 0, 0);
    return smooth::build_items(a, smooth::carve_items(reinterpret_cast<unsigned char*>(tile_state) + items_offset(B, T, N, K), B, T, N, K),
                               (cudaStream_t)stream);
}

// the items of an attention call: prepared behind the snapshots, or built now in the workspace
static int items_of(const FlashArgs& a, int flags, void* ws, smooth::Items& it, cudaStream_t st) {
    if (flags & MBEMA_FLAG_TILE_ITEMS) {
        it = smooth::carve_items(const_cast<unsigned char*>(reinterpret_cast<const unsigned char*>(a.tile_state)) + items_offset(a.B, a.T, a.N, a.K),
                                 a.B, a.T, a.N, a.K);
        return MBEMA_OK;
    }
    it = smooth::carve_items(ws, a.B, a.T, a.N, a.K);
    return smooth::build_items(a, it, st);
}

extern "C" int mbema_flash_tc_supported(int64_t H, int64_t N, int64_t K) {
    if (H < 1 || N < 1 || K < 1 || H > 65535 || K > (1 << 20)) return 0;
    return flash_tc_supported((int)H, (int)N, (int)K) ? 1 : 0;
}

static FlashArgs sizes(int64_t B, int64_t H, int64_t T, int64_t N, int64_t K) {
    return pack(nullptr, 0, nullptr, nullptr, nullptr, 0, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, B, H, T, N, K, 0, 0);
}

// the first STATUS_BYTES of a tensor-core workspace hold the kernels' status word
static constexpr size_t STATUS_BYTES = 512;

extern "C" size_t mbema_flash_fwd_workspace_bytes(int64_t B, int64_t H, int64_t T, int64_t, int64_t N, int64_t K, int mode) {
    const bool items = !(mode & MBEMA_FLAG_TILE_ITEMS);
    if ((mode & ~MBEMA_FLAG_TILE_ITEMS) == MBEMA_MODE_FP32) return flash_fwd_simt_ws(sizes(B, H, T, N, K));
    return STATUS_BYTES + smooth::ws_bytes(B, H, T, N, false) + (items ? smooth::items_bytes(B, T, N, K) : 0);
}

static int flash_fwd_impl(const void* Q, int q_dtype, const int64_t* x, const void* E_k, const void* E_v,
                          int e_dtype, const int32_t* e_row_index, int64_t e_rows, const float* W_pe, const float* rhos,
                          const int64_t* unique, const float* tile_state, const float* tok_state, const int32_t* kcount,
                          const int32_t* seq_lens, float* O, float* LSE, int64_t B, int64_t H, int64_t T,
                          int64_t hd, int64_t N, int64_t K, int64_t V_total, int flags, int mode,
                          void* workspace, size_t workspace_bytes, void* stream) {
    int rc = flash_check(B, H, T, hd, N, K, mode);
    if (rc) return rc;
    if (e_row_index && e_rows < 1) return MBEMA_ERR_SHAPE;
    if (B == 0) return MBEMA_OK;
    if (!Q || !x || !E_k || !E_v || !W_pe || !rhos || !unique || !tile_state || !tok_state || !kcount || !O || !LSE)
        return MBEMA_ERR_NULL;
    if (!dt_ok(q_dtype) || !dt_ok(e_dtype)) return MBEMA_ERR_DTYPE;
    if (((uintptr_t)Q | (uintptr_t)E_k | (uintptr_t)E_v | (uintptr_t)O | (uintptr_t)W_pe | (uintptr_t)tile_state |
         (uintptr_t)tok_state) & 15)      // all of these are read with 16-byte vector or cp.async accesses
        return MBEMA_ERR_ALIGN;
    FlashArgs a = pack(Q, q_dtype, x, E_k, E_v, e_dtype, W_pe, rhos, unique, tile_state, tok_state, kcount, seq_lens,
                       B, H, T, N, K, V_total, flags);
    a.O = O; a.LSE = LSE;
    if (e_row_index) { a.erow = e_row_index; a.e_rows = e_rows; }
    if (mode == MBEMA_MODE_TC_BF16) {
        if (!workspace) return MBEMA_ERR_NULL;
        if (workspace_bytes < mbema_flash_fwd_workspace_bytes(B, H, T, hd, N, K, mode | (flags & MBEMA_FLAG_TILE_ITEMS))) return MBEMA_ERR_WORKSPACE;
        cudaStream_t st = (cudaStream_t)stream;
        int* status = reinterpret_cast<int*>((reinterpret_cast<uintptr_t>(workspace) + 15) & ~uintptr_t(15));
        unsigned char* p = static_cast<unsigned char*>(workspace) + STATUS_BYTES;
        const smooth::Ws w = smooth::carve(p, B, H, T, N);
        smooth::Items it;
        if ((rc = items_of(a, flags, p + smooth::ws_bytes(B, H, T, N, false), it, st)) || (rc = smooth::prepare(a, it, w, st))) return rc;
        if (flags & MBEMA_FLAG_HOT_EVERY_STEP) {
            a.level = w.level;
            a.hot = it.hot;
            if ((rc = flash_fwd_tc(a, workspace, st))) return rc;
            return smooth::forward(a, it, w, status, st);
        }
        if ((rc = smooth::forward(a, it, w, status, st))) return rc;
        a.level = w.level;
        return flash_fwd_tc(a, workspace, st);
    }
    // a caller without the workspace gets the kernel that needs none
    return flash_fwd_simt(a, workspace_bytes >= flash_fwd_simt_ws(a) ? workspace : nullptr, (cudaStream_t)stream);
}

extern "C" int mbema_flash_fwd(const void* Q, int q_dtype, const int64_t* x, const void* E_k, const void* E_v,
                               int e_dtype, const float* W_pe, const float* rhos, const int64_t* unique,
                               const float* tile_state, const float* tok_state, const int32_t* kcount,
                               const int32_t* seq_lens, float* O, float* LSE, int64_t B, int64_t H, int64_t T,
                               int64_t hd, int64_t N, int64_t K, int64_t V_total, int flags, int mode,
                               void* workspace, size_t workspace_bytes, void* stream) {
    return flash_fwd_impl(Q, q_dtype, x, E_k, E_v, e_dtype, nullptr, 0, W_pe, rhos, unique, tile_state, tok_state, kcount,
                          seq_lens, O, LSE, B, H, T, hd, N, K, V_total, flags, mode, workspace, workspace_bytes, stream);
}

extern "C" int mbema_flash_fwd_rows(const void* Q, int q_dtype, const int64_t* x, const void* E_k, const void* E_v,
                                    int e_dtype, const int32_t* e_row_index, int64_t e_rows, const float* W_pe,
                                    const float* rhos, const int64_t* unique, const float* tile_state,
                                    const float* tok_state, const int32_t* kcount, const int32_t* seq_lens, float* O,
                                    float* LSE, int64_t B, int64_t H, int64_t T, int64_t hd, int64_t N, int64_t K,
                                    int64_t V_total, int flags, int mode, void* workspace, size_t workspace_bytes,
                                    void* stream) {
    if (!e_row_index) return MBEMA_ERR_NULL;
    return flash_fwd_impl(Q, q_dtype, x, E_k, E_v, e_dtype, e_row_index, e_rows, W_pe, rhos, unique, tile_state, tok_state,
                          kcount, seq_lens, O, LSE, B, H, T, hd, N, K, V_total, flags, mode, workspace, workspace_bytes,
                          stream);
}

extern "C" size_t mbema_flash_bwd_workspace_bytes(int64_t B, int64_t H, int64_t T, int64_t hd, int64_t N, int64_t K,
                                                  int mode) {
    (void)hd;
    const bool items = !(mode & MBEMA_FLAG_TILE_ITEMS);
    mode &= ~MBEMA_FLAG_TILE_ITEMS;
    // in tensor-core mode the first 512 bytes hold the kernel status word, whichever kernel ends up running
    size_t need = flash_bwd_simt_ws(sizes(B, H, T, N, K)) + (mode == MBEMA_MODE_TC_BF16 ? 512 : 0);
    if (mode == MBEMA_MODE_TC_BF16 && flash_bwd_tc_supported((int)H, (int)N, (int)K)) {
        const size_t tc = flash_bwd_tc_ws(B, H, T, N) + smooth::ws_bytes(B, H, T, N, true) + (items ? smooth::items_bytes(B, T, N, K) : 0);
        if (tc > need) need = tc;
    }
    return need;
}

static int flash_bwd_impl(const void* Q, int q_dtype, const int64_t* x, const void* E_k, const void* E_v,
                          int e_dtype, const int32_t* e_row_index, int64_t e_rows, const float* W_pe, const float* rhos,
                          const int64_t* unique, const float* tile_state, const float* tok_state, const int32_t* kcount,
                          const int32_t* seq_lens, const float* O, const float* LSE, const void* dO,
                          int do_dtype, float* dQ, float* dE_k, float* dE_v, float* dW_pe, int64_t B, int64_t H,
                          int64_t T, int64_t hd, int64_t N, int64_t K, int64_t V_total, int flags, int mode,
                          void* workspace, size_t workspace_bytes, void* stream) {
    int rc = flash_check(B, H, T, hd, N, K, mode);
    if (rc) return rc;
    if (e_row_index && e_rows < 1) return MBEMA_ERR_SHAPE;
    if (!dW_pe) return MBEMA_ERR_NULL;
    cudaStream_t st = (cudaStream_t)stream;
    if (B == 0) {
        MBEMA_CUDA_TRY(cudaMemsetAsync(dW_pe, 0, (size_t)N * H * hd * sizeof(float), st));
        return MBEMA_OK;
    }
    if (!Q || !x || !E_k || !E_v || !W_pe || !rhos || !unique || !tile_state || !tok_state || !kcount || !O || !LSE ||
        !dO || !dQ || !dE_k || !dE_v || !workspace)
        return MBEMA_ERR_NULL;
    if (!dt_ok(q_dtype) || !dt_ok(e_dtype) || !dt_ok(do_dtype)) return MBEMA_ERR_DTYPE;
    if (((uintptr_t)Q | (uintptr_t)E_k | (uintptr_t)E_v | (uintptr_t)O | (uintptr_t)dO | (uintptr_t)dQ | (uintptr_t)W_pe |
         (uintptr_t)tile_state | (uintptr_t)tok_state | (uintptr_t)dE_k | (uintptr_t)dE_v | (uintptr_t)dW_pe) & 15)
        return MBEMA_ERR_ALIGN;
    if (workspace_bytes < mbema_flash_bwd_workspace_bytes(B, H, T, hd, N, K, mode | (flags & MBEMA_FLAG_TILE_ITEMS))) return MBEMA_ERR_WORKSPACE;
    FlashArgs a = pack(Q, q_dtype, x, E_k, E_v, e_dtype, W_pe, rhos, unique, tile_state, tok_state, kcount, seq_lens,
                       B, H, T, N, K, V_total, flags);
    a.O = const_cast<float*>(O); a.LSE = const_cast<float*>(LSE);
    a.dO = dO; a.do_dt = do_dtype; a.dQ = dQ; a.dEk = dE_k; a.dEv = dE_v;
    if (e_row_index) { a.erow = e_row_index; a.e_rows = e_rows; }
    // tensor-core backward where the shape fits its shared-memory budget (N == 64); otherwise the fp32 kernels
    if (mode == MBEMA_MODE_TC_BF16) {
        if (!(flags & MBEMA_FLAG_FP32_BACKWARD) && flash_bwd_tc_supported((int)H, (int)N, (int)K)) {
            unsigned char* p = static_cast<unsigned char*>(workspace) + flash_bwd_tc_ws(B, H, T, N);
            const smooth::Ws w = smooth::carve(p, B, H, T, N);
            smooth::Items it;
            if ((rc = items_of(a, flags, p + smooth::ws_bytes(B, H, T, N, true), it, st))) return rc;
            return flash_bwd_tc(a, it, w, dW_pe, workspace, st);
        }
        // (the first 512 bytes stay reserved for the status word of the tensor-core kernels; the fp32 kernels have no
        // bounded waits and leave it alone)
        return flash_bwd_simt(a, dW_pe, static_cast<unsigned char*>(workspace) + 512, st);
    }
    return flash_bwd_simt(a, dW_pe, workspace, st);
}

extern "C" int mbema_flash_bwd(const void* Q, int q_dtype, const int64_t* x, const void* E_k, const void* E_v,
                               int e_dtype, const float* W_pe, const float* rhos, const int64_t* unique,
                               const float* tile_state, const float* tok_state, const int32_t* kcount,
                               const int32_t* seq_lens, const float* O, const float* LSE, const void* dO,
                               int do_dtype, float* dQ, float* dE_k, float* dE_v, float* dW_pe, int64_t B, int64_t H,
                               int64_t T, int64_t hd, int64_t N, int64_t K, int64_t V_total, int flags, int mode,
                               void* workspace, size_t workspace_bytes, void* stream) {
    return flash_bwd_impl(Q, q_dtype, x, E_k, E_v, e_dtype, nullptr, 0, W_pe, rhos, unique, tile_state, tok_state, kcount,
                          seq_lens, O, LSE, dO, do_dtype, dQ, dE_k, dE_v, dW_pe, B, H, T, hd, N, K, V_total, flags, mode,
                          workspace, workspace_bytes, stream);
}

extern "C" int mbema_flash_bwd_rows(const void* Q, int q_dtype, const int64_t* x, const void* E_k, const void* E_v,
                                    int e_dtype, const int32_t* e_row_index, int64_t e_rows, const float* W_pe,
                                    const float* rhos, const int64_t* unique, const float* tile_state,
                                    const float* tok_state, const int32_t* kcount, const int32_t* seq_lens,
                                    const float* O, const float* LSE, const void* dO, int do_dtype, float* dQ,
                                    float* dE_k, float* dE_v, float* dW_pe, int64_t B, int64_t H, int64_t T, int64_t hd,
                                    int64_t N, int64_t K, int64_t V_total, int flags, int mode, void* workspace,
                                    size_t workspace_bytes, void* stream) {
    if (!e_row_index) return MBEMA_ERR_NULL;
    return flash_bwd_impl(Q, q_dtype, x, E_k, E_v, e_dtype, e_row_index, e_rows, W_pe, rhos, unique, tile_state, tok_state,
                          kcount, seq_lens, O, LSE, dO, do_dtype, dQ, dE_k, dE_v, dW_pe, B, H, T, hd, N, K, V_total, flags,
                          mode, workspace, workspace_bytes, stream);
}
