// Attention over slot states that vary smoothly inside a time tile ("smooth path"): shared declarations.
//
// Between two occurrences of its token a slot's state only decays, M_n(t) = M_n(t0) rho_n^(t - t0), so with half-lives
// of hundreds of steps the gate SiLU(M(t) W) of a slot is a smooth function of t over a tile of 128 steps.  It is
// evaluated at the four Chebyshev nodes of the tile instead of at its 128 steps and expanded in the Chebyshev
// polynomials T_0..T_3 of the step: gate[t,k,d] = sum_j T_j(t) c_j[k,d].  With Q'[t,(j,d)] = T_j(t) Q[t,d] the operator
// becomes an ordinary attention with head width 4 * 64 over the virtual keys E_k c_j and values E_v c_j, all of it
// tensor-core products; one gate evaluation serves 32 steps.  An occurrence inside the tile starts a new item with the
// state (state + 1) rho^-(step), extended backwards to the tile start and valid for the steps after it.
//
// Error: with d the change of a column's pre-activation over half a segment, the cubic interpolant of SiLU is off by at most
// 1.8e-3 d^4 / (1 + 0.033 d^3) (root mean square over the segment; an upper fit of the measured error for d in 0.1 .. 12), and only
// where the column passes through the bend of SiLU, |x| < d + 3.5.  k_levels evaluates this for every item and head with the actual
// pre-activations, and picks the number of segments the tile is cut into (1, 2, 4 or 8, each with nodes of its own) so that the
// interpolation moves no item's gate by more than TOL_GATE of its norm over a head's columns; what eight segments do not resolve goes to
// the kernels that evaluate every step (level LEVEL_EXACT).  Against 64 bits the outputs are then closer than the every-step kernels':
// 5.2e-4 (2-norm) against 6.2e-4 for the 46M training chunks, W_pe ~ N(0, 0.02^2), states to 600.
#pragma once
#include "flash.cuh"
#include <cuda_fp16.h>

namespace mbema {
namespace smooth {

static constexpr int TM = MBEMA_TILE_T;     // steps per tile
static constexpr int HD = 64;
static constexpr int NJ = 4;                // nodes = coefficients per item
static constexpr int IBLK = 128;            // items per block
static constexpr int NCH = 4;               // a head's 64 columns are walked in chunks of 16: 16 x NJ = one swizzle atom
static constexpr int ATOM = TM * 128;       // bytes of a 128-row x 64-column 16-bit operand tile
static constexpr int WPIECE = 64 * 128;     // W' rows (node, 16 columns) x 64 channels
static constexpr int LEVELS = 4;            // level L cuts the tile into 2^L segments
static constexpr int LEVEL_EXACT = LEVELS;
static constexpr int SEG_IMAGES = (1 << LEVELS) - 1;   // W' images: segment s of level L at index 2^L - 1 + s
// Half a segment's decay exponent that a cubic still resolves: remainder below 0.16^4 / 192 = 3.4e-6 of the state sum.  The
// backward's two-term node powers (smooth_bwd.cu) want it smaller: 0.045^2 / 4 = 5e-4.
static constexpr float MAX_DECAY = 0.16f, MAX_DECAY_BWD = 0.045f;
// Interpolation error of an item's gate over a head's columns, relative to their norm: half the unit roundoff of the fp16 that gates
// are packed to (2^-11).  In the backward the same for SiLU' with the full unit.
static constexpr float TOL_GATE = 1.0f / 4096.0f, TOL_SLOPE = 1.0f / 2048.0f;
// Items whose pre-activations cannot change by more than this over half a tile meet TOL_GATE in every case (1.8e-3 d^4 against
// a gate that itself moves by d / 3) and are not looked at.
static constexpr float SMALL_SWING = 0.35f;
// The coefficients are sums of up to four gates in fp16: items of larger ones (norm over a head's columns at mid-tile; up to
// 3.6 times as much at the start of the fastest decays that eight segments resolve) go to the every-step kernels.
static constexpr float MAX_GATE = 4096.0f;
static constexpr float STATE_WEIGHT = 64.0f * 0.5f * MAX_GATE / SMALL_SWING;      // |state| that can reach half of it counts like a change of SMALL_SWING

// Slots with the largest states, per tile.  They stand at the end of the item list, in blocks of their own: the forward walks
// all blocks, the backward leaves these slots to the every-step kernel.  Their pre-activations move most inside a tile
// and their gradient rows are the largest of a batch (tens of times the mean), at 1 to 5 % of the work.
static constexpr int HOT = 16;

// What precompute_boundaries prepares once for all attention calls on a chunk batch: the items of every (sample, tile).
struct Items {
    unsigned char* a_img;   // [B * nT][IB][N / 64][ATOM] item states, fp16 of state / 64, swizzled operand tiles
    uint4* mask;            // [B * nT][IB][128] bit i of row t: item i of the block is valid at step t
    int2* meta;             // [B * nT][IB * 128] {slot, first valid step | last << 8}
    int* src;               // [B * nT][IB * 128] where the state comes from: slot k (snapshot) or -1 - step (occurrence); INT_MAX: padding
    float* q;               // [B * nT][IB * 128] |lambda . state|^2 (or |state|^2 / STATE_WEIGHT^2 where that is larger)
    int4* count;            // [B * nT] {items and blocks before the hot ones, items and blocks in all}
    int* hot;               // [B * nT][HOT + 1] number of hot slots, the slots
    int IB;                 // blocks reserved per tile
};

// Per-call workspace (after the status block).
struct Ws {
    __half* probe;          // [3][D][N] W_pe scaled to pre-activations at mid-tile, and to their change over half a tile at the start and the end
    float* wnorm;           // [D] |column of W_pe|^2
    unsigned char* w_img;   // [SEG_IMAGES][H][NCH][N / 64][WPIECE] node-scaled W_pe, fp16, swizzled operand pieces
    int* level;             // [B * nT] of the forward
    int* level_bwd;         // [B * nT] of the backward
    unsigned char* do_img;  // N = 128, backward: [B * nT][H][NCH][ATOM] dO' operand tiles
};

inline size_t items_bytes(int64_t B, int64_t T, int64_t N, int64_t K) {
    const size_t tiles = (size_t)B * ((T + TM - 1) / TM), IB = (size_t)(K + TM + IBLK - 1) / IBLK + 2, NK = (size_t)N / 64;
    return tiles * IB * (NK * ATOM + IBLK * (sizeof(uint4) + sizeof(int2) + sizeof(int) + sizeof(float))) + tiles * sizeof(int4) +
           tiles * (HOT + 1) * 4 + 2048;
}

inline Items carve_items(void* p0, int64_t B, int64_t T, int64_t N, int64_t K) {
    const size_t tiles = (size_t)B * ((T + TM - 1) / TM), IB = (size_t)(K + TM + IBLK - 1) / IBLK + 2, NK = (size_t)N / 64;
    unsigned char* p = reinterpret_cast<unsigned char*>(align_up(reinterpret_cast<size_t>(p0), 1024));
    Items t;
    t.IB = (int)IB;
    t.a_img = p; p += tiles * IB * NK * ATOM;
    t.mask = reinterpret_cast<uint4*>(p); p += tiles * IB * IBLK * sizeof(uint4);
    t.meta = reinterpret_cast<int2*>(p); p += tiles * IB * IBLK * sizeof(int2);
    t.count = reinterpret_cast<int4*>(p); p += tiles * sizeof(int4);
    t.src = reinterpret_cast<int*>(p); p += tiles * IB * IBLK * sizeof(int);
    t.q = reinterpret_cast<float*>(p); p += tiles * IB * IBLK * sizeof(float);
    t.hot = reinterpret_cast<int*>(p);
    return t;
}

inline size_t ws_bytes(int64_t B, int64_t H, int64_t T, int64_t N, bool backward) {
    const size_t tiles = (size_t)B * ((T + TM - 1) / TM), NK = (size_t)N / 64;
    return align_up((size_t)H * HD * (3 * N * 2 + 4), 1024) + SEG_IMAGES * (size_t)H * NCH * NK * WPIECE + 2 * align_up(tiles * 4, 1024) +
           (backward && NK == 2 ? tiles * H * NCH * ATOM : 0) + 1024;
}

inline Ws carve(void* p0, int64_t B, int64_t H, int64_t T, int64_t N) {
    const size_t tiles = (size_t)B * ((T + TM - 1) / TM), NK = (size_t)N / 64;
    unsigned char* p = reinterpret_cast<unsigned char*>(align_up(reinterpret_cast<size_t>(p0), 1024));
    Ws w;
    w.probe = reinterpret_cast<__half*>(p);
    w.wnorm = reinterpret_cast<float*>(p + (size_t)H * HD * 3 * N * 2); p += align_up((size_t)H * HD * (3 * N * 2 + 4), 1024);
    w.w_img = p; p += SEG_IMAGES * (size_t)H * NCH * NK * WPIECE;
    w.level = reinterpret_cast<int*>(p); p += align_up(tiles * 4, 1024);
    w.level_bwd = reinterpret_cast<int*>(p); p += align_up(tiles * 4, 1024);
    w.do_img = p;
    return w;
}

// Chebyshev basis of a step, scaled so that the coefficients need no factors: beta_j = s_j T_j(u) with
// s = {1, 2 cos(pi/8), sqrt 2, -2 cos(pi/8)}, the E rows taken times 1/4 and the coefficients formed as
//   c_0 = (g0 + g3) + (g1 + g2)   c_1 = (g0 - g3) + tan(pi/8) (g1 - g2)   c_2 = (g0 + g3) - (g1 + g2)   c_3 = (g1 - g2) - tan(pi/8) (g0 - g3)
__device__ __forceinline__ void basis(int row, int level, float (&beta)[NJ]) {
    const int len = TM >> level;
    const float u = ((float)(row & (len - 1)) - 0.5f * (float)(len - 1)) * (2.0f / (float)len);
    const float t2 = fmaf(2.0f * u, u, -1.0f);
    beta[0] = 1.0f;
    beta[1] = 1.8477590650f * u;
    beta[2] = 1.4142135624f * t2;
    beta[3] = -1.8477590650f * u * fmaf(2.0f, t2, -1.0f);     // T_3 = u (4 u^2 - 3) = u (2 T_2 - 1)
}
static constexpr float TAN_PI_8 = 0.41421356237f;

// items of a chunk batch (a: x, unique, rhos, tile_state, tok_state, kcount, seq_lens and the sizes)
int build_items(const FlashArgs& a, const Items& it, cudaStream_t st);
// what depends on W_pe: node-scaled images, levels
int prepare(const FlashArgs& a, const Items& it, const Ws& w, cudaStream_t st);
int forward(const FlashArgs& a, const Items& it, const Ws& w, int* status, cudaStream_t st);
int backward(const FlashArgs& a, const Items& it, const Ws& w, int* status, cudaStream_t st);

}  // namespace smooth
}  // namespace mbema
