// K3: reverse-mode (adjoint) Euler step of the Fenton-Karma stepper.
//
// Forward step (cardiax/solve.py:26-70), per cell:  v' = v + dt dv,  w' = w + dt dw,
// u' = u + dt (L(D) u + J), with J replaced by the stimulus value where one is active and
// L(D) u = D (A_x + A_y) u + (B_x D)(B_x u) + (B_y D)(B_y u).  Along one axis of length N,
// with E the edge pad (N+2 x N), G the derivative of cardiax/solve.py:225-254 on the padded
// line and C the crop:  B = C G E / dx,  A = C G G E / dx^2.
//
// Given the state x_t and the cotangent lam' of x_{t+1}, this computes the cotangent of x_t,
//   lam_v = lam'_v dv'/dv + lam'_u dt dJ/dv,   lam_w = lam'_w dw'/dw + lam'_u dt dJ/dw,
//   lam_u = lam'_u (1 + dt dJ/du) + L^T mu,     mu = dt lam'_u,
//   L^T mu = A_x^T (D mu) + A_y^T (D mu) + B_x^T ((B_x D) mu) + B_y^T ((B_y D) mu),
// and accumulates  dL/dD += mu (u_xx + u_yy) + B_x^T (mu u_x) + B_y^T (mu u_y)  per cell and
// dL/dtheta for the first 13 parameters (Cm fixed).  The Heaviside gates have zero derivative
// and a stimulated cell's J does not depend on the state or theta, exactly as jnp.where and
// jnp.greater_equal differentiate in the reference.
//
// Interior cells use G^T = -G on central rows (so A^T = A and B^T = -B); cells within
// ADJ_BAND of an edge use the explicit transposed rows, including the one-sided rows and the
// fold of the edge pad.
#include <cuda_runtime.h>

#include <cstdint>

#include "fk_adjoint.cuh"
#include "fk_capi_internal.h"
#include "fk_math.cuh"
#include "fk_pack.cuh"
#include "fk_ptx.cuh"

namespace fk {

namespace {

__device__ __forceinline__ int clampi(int x, int lo, int hi) { return x < lo ? lo : (x > hi ? hi : x); }

// Coefficient of P[m] in row k of G on a padded line of length L (cardiax/solve.py:225-254).
__device__ __forceinline__ float gcoef(int k, int m, int L) {
    int o;
    if (k < 2) {  // head rows: P[k..k+3]
        o = m - k;
        switch (o) {
            case 0: return C_HEAD0;
            case 1: return C_THREE;
            case 2: return -C_3_2;
            case 3: return C_1_3;
            default: return 0.0f;
        }
    }
    if (k > L - 3) {  // tail rows: P[k-3..k]
        o = m - (k - 3);
        switch (o) {
            case 0: return C_TAIL0;
            case 1: return C_3_2;
            case 2: return -C_THREE;
            case 3: return C_TAIL3;
            default: return 0.0f;
        }
    }
    o = m - k;  // central rows: P[k-2], P[k-1], P[k+1], P[k+2]
    switch (o) {
        case -2: return C_1_12;
        case -1: return -C_2_3;
        case 1: return C_2_3;
        case 2: return -C_1_12;
        default: return 0.0f;
    }
}

// Accessor of a field along one line (a row or a column of the grid) at interior index r.
template <class F>
struct Line {
    F f;
    int N;
    // z = C^T a: padded index k -> a(k-1) for 1 <= k <= N, 0 at the pad
    __device__ __forceinline__ float z(int k) const { return (k >= 1 && k <= N) ? f(k - 1) : 0.0f; }
    // y1 = G^T z at padded index m
    __device__ float y1(int m) const {
        const int L = N + 2;
        float s = 0.0f;
        for (int k = max(0, m - 4); k <= min(L - 1, m + 4); ++k) {
            const float c = gcoef(k, m, L);
            if (c != 0.0f) s = fmaf(c, z(k), s);
        }
        return s;
    }
    // y2 = G^T y1 at padded index m
    __device__ float y2(int m) const {
        const int L = N + 2;
        float s = 0.0f;
        for (int k = max(0, m - 4); k <= min(L - 1, m + 4); ++k) {
            const float c = gcoef(k, m, L);
            if (c != 0.0f) s = fmaf(c, y1(k), s);
        }
        return s;
    }
    // (E^T y)[i]: the pad rows fold back onto the first and last cells
    __device__ float BT(int i) const {
        float s = y1(i + 1);
        if (i == 0) s += y1(0);
        if (i == N - 1) s += y1(N + 1);
        return s;
    }
    __device__ float AT(int i) const {
        float s = y2(i + 1);
        if (i == 0) s += y2(0);
        if (i == N - 1) s += y2(N + 1);
        return s;
    }
};

template <class F>
__device__ __forceinline__ Line<F> make_line(F f, int N) {
    return Line<F>{f, N};
}

// Forward first derivative (scaled by 1/dx later) at interior index i along a line accessed
// with clamped indices (the edge pad), as in the forward kernels' boundary path.
template <class F>
__device__ __forceinline__ float fwd_d1(F at, int i, int N) {
    // padded index i+1 of the derivative of the padded line
    const int x = i;
    if (x <= 0) return g_head(at(x), at(x + 1), at(x + 2), at(x + 3));
    if (x >= N - 1) return g_tail(at(x - 3), at(x - 2), at(x - 1), at(x));
    return g_central(at(x - 2), at(x - 1), at(x + 1), at(x + 2));
}
// u_x on the padded line at padded position x in [-1, N] (the first derivative that the
// second derivative is taken of).
template <class F>
__device__ __forceinline__ float fwd_ux_pad(F at, int x, int N) {
    if (x <= 0) return g_head(at(x), at(x + 1), at(x + 2), at(x + 3));
    if (x >= N - 1) return g_tail(at(x - 3), at(x - 2), at(x - 1), at(x));
    return g_central(at(x - 2), at(x - 1), at(x + 1), at(x + 2));
}
template <class F>
__device__ __forceinline__ float fwd_d2(F at, int i, int N, float rdx) {
    auto UX = [&](int x) { return fwd_ux_pad(at, x, N) * rdx; };
    float s;
    if (i == 0) s = g_head(UX(0), UX(1), UX(2), UX(3));
    else if (i == N - 1) s = g_tail(UX(N - 4), UX(N - 3), UX(N - 2), UX(N - 1));
    else s = g_central(UX(i - 2), UX(i - 1), UX(i + 1), UX(i + 2));
    return s * rdx;
}

// Pointwise part of the adjoint of one cell: cotangents through the gates and currents, and the
// cell's contribution to dL/dtheta (added into gth).  Returns mu = dt lam'_u.
__device__ __forceinline__ float adjoint_pointwise(const AdjointArgs &a, int i, int j, int64_t off,
                                                  float &olv, float &olw, float &olu,
                                                  float *gth) {
    const Model &m = a.m;
    const float dt = a.dt;
    const float u = __ldg(a.u + off), v = __ldg(a.v + off), w = __ldg(a.w + off);
    const float lu = __ldg(a.lu + off), lv = __ldg(a.lv + off), lw = __ldg(a.lw + off);
    const float mu = dt * lu;
    bool stim = false;
    for (int s = 0; s < a.n_stim; ++s) {
        if (!stim_active(a.stim[s], a.t)) continue;
        const Stim &st = a.stim[s];
        const float fv = st.field ? __ldg(st.field + off)
                                  : ((i >= st.r0 && i < st.r1 && j >= st.c0 && j < st.c1)
                                         ? st.amplitude : 0.0f);
        if (fv != 0.0f) stim = true;
    }
    const bool p = u >= m.V_c, q = u >= m.V_v;
    const float S = one_plus_tanh(m.k * (u - m.V_csi));  // 1 + tanh
    const float sech2 = S * (2.0f - S);                  // 1 - tanh^2
    const float r_tvm = q ? m.r_tau_v2m : m.r_tau_v1m;
    const float dvdv = 1.0f + dt * (p ? -m.r_tau_vp : -r_tvm);
    const float dwdw = 1.0f + dt * (p ? -m.r_tau_wp : -m.r_tau_wm);
    float dJdu = 0.f, dJdv = 0.f, dJdw = 0.f;
    if (!stim) {
        const float dfi = p ? -v * (1.0f + m.V_c - 2.0f * u) * m.r_tau_d : 0.0f;
        const float dso = p ? 0.0f : m.r_tau_0;
        const float dsi = -w * m.k * sech2 * m.r_2tau_si;
        dJdu = -(dfi + dso + dsi) * m.r_Cm;
        dJdv = p ? (u - m.V_c) * (1.0f - u) * m.r_tau_d * m.r_Cm : 0.0f;
        dJdw = S * m.r_2tau_si * m.r_Cm;
    }
    olv = lv * dvdv + mu * dJdv;
    olw = lw * dwdw + mu * dJdw;
    olu = lu * (1.0f + dt * dJdu);

    // parameter gradients (cardiax/params.py fields 0..12)
    const float pv = p ? 1.0f : 0.0f, qv = q ? 1.0f : 0.0f;
    gth[0] += lv * dt * pv * v * m.r_tau_vp * m.r_tau_vp;                           // tau_v_plus
    gth[1] += -lv * dt * (1.f - pv) * (1.f - v) * (1.f - qv) * m.r_tau_v1m * m.r_tau_v1m;
    gth[2] += -lv * dt * (1.f - pv) * (1.f - v) * qv * m.r_tau_v2m * m.r_tau_v2m;
    gth[3] += lw * dt * pv * w * m.r_tau_wp * m.r_tau_wp;                           // tau_w_plus
    gth[4] += -lw * dt * (1.f - pv) * (1.f - w) * m.r_tau_wm * m.r_tau_wm;           // tau_w_minus
    if (!stim) {
        gth[5] += mu * (-v * pv * (u - m.V_c) * (1.f - u) * m.r_tau_d * m.r_tau_d) * m.r_Cm;
        gth[6] += mu * (u * (1.f - pv) * m.r_tau_0 * m.r_tau_0) * m.r_Cm;            // tau_0
        gth[7] += mu * (pv * m.inv_tau_r * m.inv_tau_r) * m.r_Cm;                    // tau_r
        gth[8] += mu * (-w * S * 2.0f * m.r_2tau_si * m.r_2tau_si) * m.r_Cm;         // tau_si
        gth[9] += mu * (w * sech2 * (u - m.V_csi) * m.r_2tau_si) * m.r_Cm;           // k
        gth[10] += mu * (-w * m.k * sech2 * m.r_2tau_si) * m.r_Cm;                   // V_csi
        gth[11] += mu * (-v * pv * (1.f - u) * m.r_tau_d) * m.r_Cm;                  // V_c
    }
    // gth[12] (V_v) enters only through a Heaviside gate: zero
    return mu;
}

// One axis of the diffusion transpose at a cell within ADJ_BAND of an edge along that axis:
// the explicit transposed rows (one-sided rows and the fold of the edge pad), reading global
// memory.  AXIS 0: along rows (x), 1: along columns (y).
struct AxisTerms {
    float AT, BT, d2, g;  // A^T(D mu), B^T((B D) mu), u_xx (or u_yy), B^T(mu u_x) (or y)
};
template <int AXIS>
__device__ AxisTerms axis_explicit(const AdjointArgs &a, int i, int j) {
    const int H = a.H, W = a.W, pitch = a.pitch;
    const float dt = a.dt, rdx = a.rdx;
    const float *D = a.D, *U = a.u, *LU = a.lu;
    auto at = [&](const float *p, int r, int c) {
        return __ldg(p + (int64_t)clampi(r, 0, H - 1) * pitch + clampi(c, 0, W - 1));
    };
    AxisTerms t;
    if (AXIS == 0) {
        auto Dx_at = [&](int r) { return fwd_d1([&](int x) { return at(D, x, j); }, r, H) * rdx; };
        auto Ux_at = [&](int r) { return fwd_d1([&](int x) { return at(U, x, j); }, r, H) * rdx; };
        auto Mcol = [&](int r) { return dt * __ldg(LU + (int64_t)r * pitch + j); };
        const auto qx = make_line([&](int r) { return at(D, r, j) * Mcol(r); }, H);
        const auto bx = make_line([&](int r) { return Dx_at(r) * Mcol(r); }, H);
        const auto gxl = make_line([&](int r) { return Mcol(r) * Ux_at(r); }, H);
        t.AT = qx.AT(i) * (rdx * rdx);
        t.BT = bx.BT(i) * rdx;
        t.d2 = fwd_d2([&](int r) { return at(U, r, j); }, i, H, rdx);
        t.g = gxl.BT(i) * rdx;
    } else {
        auto Dy_at = [&](int c) { return fwd_d1([&](int y) { return at(D, i, y); }, c, W) * rdx; };
        auto Uy_at = [&](int c) { return fwd_d1([&](int y) { return at(U, i, y); }, c, W) * rdx; };
        auto Mrow = [&](int c) { return dt * __ldg(LU + (int64_t)i * pitch + c); };
        const auto qy = make_line([&](int c) { return at(D, i, c) * Mrow(c); }, W);
        const auto by = make_line([&](int c) { return Dy_at(c) * Mrow(c); }, W);
        const auto gyl = make_line([&](int c) { return Mrow(c) * Uy_at(c); }, W);
        t.AT = qy.AT(j) * (rdx * rdx);
        t.BT = by.BT(j) * rdx;
        t.d2 = fwd_d2([&](int c) { return at(U, i, c); }, j, W, rdx);
        t.g = gyl.BT(j) * rdx;
    }
    return t;
}

// Corner blocks (cells 0..9 of a line) of the line operators B' = C G E and A' = C G G E
// (E the edge pad, G the padded-line derivative of cardiax/solve.py:225-254, C the crop), built
// in double at compile time on a line of 40 cells.  Both operators are banded (|r - i| <= 4),
// so the corner is the same for every line of at least 18 cells, and the far corner is the
// reflection: A'[N-1-r][N-1-i] = A'[r][i], B'[N-1-r][N-1-i] = -B'[r][i].
struct EdgeTables {
    float A[10][10], B[10][10];
};
constexpr double gd(int k, int m, int L) {  // G[k][m] on a padded line of length L
    if (k < 2) {
        const int o = m - k;
        return o == 0 ? -11.0 / 6.0 : o == 1 ? 3.0 : o == 2 ? -1.5 : o == 3 ? 1.0 / 3.0 : 0.0;
    }
    if (k > L - 3) {
        const int o = m - (k - 3);
        return o == 0 ? -1.0 / 3.0 : o == 1 ? 1.5 : o == 2 ? -3.0 : o == 3 ? 11.0 / 6.0 : 0.0;
    }
    const int o = m - k;
    return o == -2 ? 1.0 / 12.0 : o == -1 ? -2.0 / 3.0 : o == 1 ? 2.0 / 3.0 : o == 2 ? -1.0 / 12.0 : 0.0;
}
constexpr double ge(int m, int i, int N) {  // (G E)[m][i]
    const int L = N + 2;
    return gd(m, i + 1, L) + (i == 0 ? gd(m, 0, L) : 0.0) + (i == N - 1 ? gd(m, L - 1, L) : 0.0);
}
constexpr EdgeTables make_edge_tables() {
    constexpr int N = 40, L = N + 2;
    EdgeTables t{};
    for (int r = 0; r < 10; ++r)
        for (int i = 0; i < 10; ++i) {
            double a = 0.0;
            for (int m = 0; m < L; ++m) a += gd(r + 1, m, L) * ge(m, i, N);
            t.A[r][i] = (float)a;
            t.B[r][i] = (float)ge(r + 1, i, N);
        }
    return t;
}
constexpr EdgeTables kEdgeHost = make_edge_tables();
__constant__ EdgeTables kEdge = kEdgeHost;
constexpr int kEdgeMinLine = 20;  // shorter lines use the explicit rows of axis_explicit

// One axis of the diffusion transpose at a cell within ADJ_BAND of an end of its line, from
// the corner tables: 10 cells of the line nearest that end.
template <int AXIS>
__device__ AxisTerms axis_edge(const AdjointArgs &a, int i, int j) {
    const int N = AXIS == 0 ? a.H : a.W;
    const int pos = AXIS == 0 ? i : j;
    if (N < kEdgeMinLine) return axis_explicit<AXIS>(a, i, j);
    const int pitch = a.pitch;
    const float dt = a.dt, rdx = a.rdx;
    const bool near0 = pos < ADJ_BAND;
    const int pp = near0 ? pos : N - 1 - pos;  // distance from the near end
    auto at = [&](const float *f, int q) {
        q = clampi(q, 0, N - 1);
        return __ldg(f + (AXIS == 0 ? (int64_t)q * pitch + j : (int64_t)i * pitch + q));
    };
    float AT = 0.f, BT = 0.f, d2 = 0.f, g = 0.f;
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        const int q = near0 ? r : N - 1 - r;
        const float mu = dt * at(a.lu, q);
        const float dq = fwd_d1([&](int x) { return at(a.D, x); }, q, N) * rdx;
        const float uq = fwd_d1([&](int x) { return at(a.u, x); }, q, N) * rdx;
        AT = fmaf(kEdge.A[r][pp], at(a.D, q) * mu, AT);
        BT = fmaf(kEdge.B[r][pp], dq * mu, BT);
        d2 = fmaf(kEdge.A[pp][r], at(a.u, q), d2);
        g = fmaf(kEdge.B[r][pp], mu * uq, g);
    }
    const float sgn = near0 ? 1.0f : -1.0f;
    AxisTerms t;
    t.AT = AT * (rdx * rdx);
    t.BT = sgn * BT * rdx;
    t.d2 = d2 * (rdx * rdx);
    t.g = sgn * g * rdx;
    return t;
}

// axis_edge from a line's precomputed products (L[r] = (D mu, (B D) mu, u, mu u_x) at the r-th
// cell from the near end) and the corner tables in shared memory: the same fused multiply-adds
// in the same order, so the same bits.
__device__ __forceinline__ AxisTerms axis_edge_tab(const float4 *L, const float (*tA)[10],
                                                   const float (*tB)[10], int pp, bool near0,
                                                   float rdx) {
    float AT = 0.f, BT = 0.f, d2 = 0.f, g = 0.f;
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        const float4 l = L[r];
        AT = fmaf(tA[r][pp], l.x, AT);
        BT = fmaf(tB[r][pp], l.y, BT);
        d2 = fmaf(tA[pp][r], l.z, d2);
        g = fmaf(tB[r][pp], l.w, g);
    }
    const float sgn = near0 ? 1.0f : -1.0f;
    AxisTerms t;
    t.AT = AT * (rdx * rdx);
    t.BT = sgn * BT * rdx;
    t.d2 = d2 * (rdx * rdx);
    t.g = sgn * g * rdx;
    return t;
}

// Tile geometry: ATY x ATX cells per block, a 4-cell halo of u, D and mu in shared memory.
constexpr int ATX = 32, ATY = 16, AHALO = 4;
constexpr int ASW = ATX + 2 * AHALO, ASH = ATY + 2 * AHALO;
constexpr int ANT = 256;
constexpr int AXW = ATX;      // row width of the x-derivative planes (tile rows -2 .. ATY+1)
constexpr int AYW = ATX + 4;  // row width of the y-derivative planes (tile columns -2 .. ATX+1)

// Interior cells (at least ADJ_BAND from both ends of an axis) use G^T = -G on central rows:
// along x, A_x^T(D mu) = G G (D mu) / dx^2, B_x^T(D_x mu) = -G (D_x mu) / dx and
// B_x^T(mu u_x) = -G (mu u_x) / dx, from first derivatives staged in shared memory.
// Tile (bx, by) of the step described by `a` (a kernel parameter, or a block's shared copy);
// its dL/dtheta partial sums go to slot by * nbx + bx of a.gtheta.
__device__ __forceinline__ void adjoint_tile(const AdjointArgs &a, int bx, int by, int nbx) {
    // u, D, mu = dt lam'_u (16-byte aligned: filled with float4 stores when the halo is in-grid)
    __shared__ __align__(16) float su[ASH * ASW];
    __shared__ __align__(16) float sd[ASH * ASW];
    __shared__ __align__(16) float sm[ASH * ASW];
    __shared__ float sux[(ATY + 4) * AXW], sqx[(ATY + 4) * AXW], sbx[(ATY + 4) * AXW];
    __shared__ float suy[ATY * AYW], sqy[ATY * AYW], sby[ATY * AYW];
    __shared__ float red[kAdjParams][ANT / 32];
    // edge band: per line and end, the 10 products each band cell of that line needs (ex: the
    // x-direction lines of the tile's columns, ey: the y-direction lines of its rows), and the
    // corner tables (lanes of a column band index them with different pp)
    __shared__ float4 ex[2][ATX][10], ey[2][ATY][10];
    __shared__ float tA[10][10], tB[10][10];
    const int tid = threadIdx.x;
    const int H = a.H, W = a.W, pitch = a.pitch;
    const float dt = a.dt, rdx = a.rdx;
    const int i0 = by * ATY, j0 = bx * ATX;
    // which line ends have the cells their products read -- -1 .. 11 from the near end, the pad
    // cell included (a clamped copy in the halo) -- inside the shared halo (uniform per block)
    const bool tx0 = H >= kEdgeMinLine && i0 == 0;
    const bool tx1 = H >= kEdgeMinLine && i0 + ATY > H - ADJ_BAND && i0 <= H - 8 && i0 + ATY + 3 >= H;
    const bool ty0 = W >= kEdgeMinLine && j0 == 0;
    const bool ty1 = W >= kEdgeMinLine && j0 + ATX > W - ADJ_BAND && j0 <= W - 8 && j0 + ATX + 3 >= W;

    // u, D, mu with a 4-cell halo; out-of-grid positions hold clamped copies, read only by
    // cells that take the explicit path along that axis
    if (i0 >= AHALO && i0 + ATY + AHALO <= H && j0 >= AHALO && j0 + ATX + AHALO <= W) {
        // halo inside the grid: 16-byte loads (rows start at column j0 - 4, a multiple of 4)
        constexpr int SW4 = ASW / 4;
        for (int k = tid; k < ASH * SW4; k += ANT) {
            const int r = k / SW4, c4 = k % SW4;
            const int64_t g = (int64_t)(i0 - AHALO + r) * pitch + j0 - AHALO + 4 * c4;
            const float4 u4 = __ldg(reinterpret_cast<const float4 *>(a.u + g));
            const float4 d4 = __ldg(reinterpret_cast<const float4 *>(a.D + g));
            const float4 l4 = __ldg(reinterpret_cast<const float4 *>(a.lu + g));
            reinterpret_cast<float4 *>(su)[k] = u4;
            reinterpret_cast<float4 *>(sd)[k] = d4;
            reinterpret_cast<float4 *>(sm)[k] =
                make_float4(dt * l4.x, dt * l4.y, dt * l4.z, dt * l4.w);
        }
    } else {
        for (int k = tid; k < ASH * ASW; k += ANT) {
            const int r = k / ASW, c = k % ASW;
            const int64_t g = (int64_t)clampi(i0 - AHALO + r, 0, H - 1) * pitch +
                              clampi(j0 - AHALO + c, 0, W - 1);
            su[k] = __ldg(a.u + g);
            sd[k] = __ldg(a.D + g);
            sm[k] = dt * __ldg(a.lu + g);
        }
    }
    __syncthreads();
    // edge-band line products from the shared halo (edge tiles only)
    if (tx0 || tx1 || ty0 || ty1) {
        for (int k = tid; k < 200; k += ANT) {
            const int r = k / 10, c = k % 10;
            if (r < 10) tA[r][c] = kEdge.A[r][c];
            else tB[r - 10][c] = kEdge.B[r - 10][c];
        }
        const int nx = (tx0 + tx1) * ATX * 10, ny = (ty0 + ty1) * ATY * 10;
        for (int k = tid; k < nx + ny; k += ANT) {
            if (k < nx) {
                const int e = (!tx0 || k >= ATX * 10) ? 1 : 0;
                const int kk = k - (tx0 && e == 1 ? ATX * 10 : 0);
                const int c = kk / 10, r = kk % 10;
                const int q = e ? H - 1 - r : r;
                auto SR = [&](const float *f, int x) { return f[(x - i0 + AHALO) * ASW + c + AHALO]; };
                const float mu = SR(sm, q);
                const float dq = fwd_d1([&](int x) { return SR(sd, x); }, q, H) * rdx;
                const float uq = fwd_d1([&](int x) { return SR(su, x); }, q, H) * rdx;
                ex[e][c][r] = make_float4(SR(sd, q) * mu, dq * mu, SR(su, q), mu * uq);
            } else {
                const int k2 = k - nx;
                const int e = (!ty0 || k2 >= ATY * 10) ? 1 : 0;
                const int kk = k2 - (ty0 && e == 1 ? ATY * 10 : 0);
                const int rr = kk / 10, r = kk % 10;
                const int q = e ? W - 1 - r : r;
                auto SC = [&](const float *f, int y) { return f[(rr + AHALO) * ASW + y - j0 + AHALO]; };
                const float mu = SC(sm, q);
                const float dq = fwd_d1([&](int y) { return SC(sd, y); }, q, W) * rdx;
                const float uq = fwd_d1([&](int y) { return SC(su, y); }, q, W) * rdx;
                ey[e][rr][r] = make_float4(SC(sd, q) * mu, dq * mu, SC(su, q), mu * uq);
            }
        }
    }
    // x: u_x, G_x(D mu), D_x mu on tile rows -2 .. ATY+1
    for (int k = tid; k < (ATY + 4) * AXW; k += ANT) {
        const int r = k / AXW, c = k % AXW;
        const int b = (r - 2 + AHALO) * ASW + c + AHALO;
        auto U = [&](int d) { return su[b + d * ASW]; };
        auto Dd = [&](int d) { return sd[b + d * ASW]; };
        auto M = [&](int d) { return sm[b + d * ASW]; };
        sux[k] = g_central(U(-2), U(-1), U(1), U(2)) * rdx;
        sqx[k] = g_central(Dd(-2) * M(-2), Dd(-1) * M(-1), Dd(1) * M(1), Dd(2) * M(2)) * rdx;
        sbx[k] = (g_central(Dd(-2), Dd(-1), Dd(1), Dd(2)) * rdx) * M(0);
    }
    // y: the same on tile columns -2 .. ATX+1
    for (int k = tid; k < ATY * AYW; k += ANT) {
        const int r = k / AYW, c = k % AYW;
        const int b = (r + AHALO) * ASW + c - 2 + AHALO;
        auto U = [&](int d) { return su[b + d]; };
        auto Dd = [&](int d) { return sd[b + d]; };
        auto M = [&](int d) { return sm[b + d]; };
        suy[k] = g_central(U(-2), U(-1), U(1), U(2)) * rdx;
        sqy[k] = g_central(Dd(-2) * M(-2), Dd(-1) * M(-1), Dd(1) * M(1), Dd(2) * M(2)) * rdx;
        sby[k] = (g_central(Dd(-2), Dd(-1), Dd(1), Dd(2)) * rdx) * M(0);
    }
    __syncthreads();

    float gth[kAdjParams];
#pragma unroll
    for (int k = 0; k < kAdjParams; ++k) gth[k] = 0.0f;
    for (int k = tid; k < ATY * ATX; k += ANT) {
        const int r = k / ATX, c = k % ATX;
        const int i = i0 + r, j = j0 + c;
        if (i >= H || j >= W) continue;
        const int64_t off = (int64_t)i * pitch + j;
        float olv, olw, olu;
        const float mu = adjoint_pointwise(a, i, j, off, olv, olw, olu, gth);
        AxisTerms x, y;
        if (i >= ADJ_BAND && i < H - ADJ_BAND) {
            auto X = [&](const float *f, int d) { return f[(r + 2 + d) * AXW + c]; };
            auto M = [&](int d) { return sm[(r + AHALO + d) * ASW + c + AHALO]; };
            x.AT = g_central(X(sqx, -2), X(sqx, -1), X(sqx, 1), X(sqx, 2)) * rdx;
            x.BT = -g_central(X(sbx, -2), X(sbx, -1), X(sbx, 1), X(sbx, 2)) * rdx;
            x.d2 = g_central(X(sux, -2), X(sux, -1), X(sux, 1), X(sux, 2)) * rdx;
            x.g = -g_central(M(-2) * X(sux, -2), M(-1) * X(sux, -1), M(1) * X(sux, 1),
                             M(2) * X(sux, 2)) * rdx;
        } else {
            const bool near0 = i < ADJ_BAND;
            if (near0 ? tx0 : tx1)
                x = axis_edge_tab(ex[near0 ? 0 : 1][c], tA, tB, near0 ? i : H - 1 - i, near0, rdx);
            else
                x = axis_edge<0>(a, i, j);
        }
        if (j >= ADJ_BAND && j < W - ADJ_BAND) {
            auto Y = [&](const float *f, int d) { return f[r * AYW + c + 2 + d]; };
            auto M = [&](int d) { return sm[(r + AHALO) * ASW + c + AHALO + d]; };
            y.AT = g_central(Y(sqy, -2), Y(sqy, -1), Y(sqy, 1), Y(sqy, 2)) * rdx;
            y.BT = -g_central(Y(sby, -2), Y(sby, -1), Y(sby, 1), Y(sby, 2)) * rdx;
            y.d2 = g_central(Y(suy, -2), Y(suy, -1), Y(suy, 1), Y(suy, 2)) * rdx;
            y.g = -g_central(M(-2) * Y(suy, -2), M(-1) * Y(suy, -1), M(1) * Y(suy, 1),
                             M(2) * Y(suy, 2)) * rdx;
        } else {
            const bool near0 = j < ADJ_BAND;
            if (near0 ? ty0 : ty1)
                y = axis_edge_tab(ey[near0 ? 0 : 1][r], tA, tB, near0 ? j : W - 1 - j, near0, rdx);
            else
                y = axis_edge<1>(a, i, j);
        }
        const float diff_u = (x.AT + y.AT) + (x.BT + y.BT);
        const float gD = mu * (x.d2 + y.d2) + (x.g + y.g);
        a.olv[off] = olv;
        a.olw[off] = olw;
        a.olu[off] = olu + diff_u;
        if (a.gD) a.gD[off] += gD;
    }

    // ---- deterministic block reduction of the parameter gradients into this block's slot ----
    if (a.gtheta) {
        const int lane = tid & 31, warp = tid >> 5;
#pragma unroll
        for (int k = 0; k < kAdjParams; ++k) {
            float x = gth[k];
            for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
            if (lane == 0) red[k][warp] = x;
        }
        __syncthreads();
        if (tid < kAdjParams) {
            double s = 0.0;
            for (int w = 0; w < ANT / 32; ++w) s += (double)red[tid][w];
            a.gtheta[(int64_t)(by * nbx + bx) * kAdjParamStride + tid] += s;
        }
    }
}

__global__ void __launch_bounds__(ANT, 4) fk_adjoint_kernel(const __grid_constant__ AdjointArgs a) {
    adjoint_tile(a, blockIdx.x, blockIdx.y, gridDim.x);
}

// ---- lines of at least kLineMin cells: two or four threads per unit of two rows of a quad ----------
// What bounds it: the tile kernel above stages six derivative planes, tests every stimulus's protocol in every
// cell and reduces 13 parameter sums over a warp for every two cells (us per step: 39.5 for 16 experiments of
// 256^2, 10.9 for one 151 x 203 grid, 10.5 for 16 of 64^2).  Here everything comes from one staged tile of u, D
// and lambda_u and stays in registers: 24.7, 5.0 and 5.2 us.  Many experiments are bound by the instructions of the
// stencils and currents; one small grid waits for its launch (4 us without any work) and then for the longest
// chain of a unit.
//   * lambda and dL/dD are the tile kernel's operations in the same order: the same bits.  (Regrouped, the two
//     products of an axis sharing their second operator and the one-sided rows as rank-one terms, the step took
//     24.1, 5.1 and 6.1 us; but rounding at the edges acts the same way in every step, and dL/dw0 of small grids
//     came out up to 3.8 times further from the 64-bit gradient.)  Along columns four lines are two packed
//     operations.
//   * cells within ADJ_BAND of a line's end: the ten products at that end once per line, then one thread per
//     cell and line sums them with the corner tables; the units take all other cells by the central operators
//     alone, so that no warp goes two ways.
//   * the constant factors of the parameter sums are applied once, in double, to sums that are reduced over a
//     warp once per 8 cells.
constexpr int kLineMin = kEdgeMinLine;  // shorter lines (fewer than three quads or nine rows in a last tile)
                                        // take the tile kernel above
constexpr int LR = 2;         // rows per thread
constexpr int LG = 8;         // most row groups of a tile
constexpr int LROWS = LG * LR;
constexpr int LNT = 256;      // threads of a block: two or four share a unit (see fk_adjoint_line_kernel)
constexpr int LEND = 10;      // cells at a line's end that the band's sums take
template <int SHARE>
struct LineTile {
    static constexpr int LU = LNT / SHARE, LQ = LU / LG;  // units, most quads of a tile
    static constexpr int LSW = 4 * LQ + 12;  // staged row: 4 cells on either side, and 4 more so that 8 lanes
                                             // (2 quads of 4 groups) read from 8 different 16-byte banks
    static constexpr int LSH = LROWS + 8 + 1;  // 4 rows above and below; the first group of the last
                                               // tile row may reach one row further up
    static constexpr int LC = 4 * LQ;          // columns
    static constexpr int SMEM = (3 * LSH * LSW + 8 * LR * LU * 4 +
                                 4 * (LEND * LC + 2 * LEND * LROWS + 2 * ADJ_BAND * LROWS + LEND * ADJ_BAND)) * 4;
};

// The corner tables by what a cell `pp` from the line's end takes of cell r: A[r][pp], B[r][pp], A[pp][r].
struct alignas(16) EndTap {
    float a, b, d, pad;
};
struct EndTaps {
    EndTap t[LEND][ADJ_BAND];
};
constexpr EndTaps make_end_taps() {
    EndTaps x{};
    for (int r = 0; r < LEND; ++r)
        for (int p = 0; p < ADJ_BAND; ++p)
            x.t[r][p] = EndTap{kEdgeHost.A[r][p], kEdgeHost.B[r][p], kEdgeHost.A[p][r], 0.0f};
    return x;
}
__device__ const EndTaps kEndTaps = make_end_taps();

// D mu, (B D) mu, u and mu u' at the cell at place b of the staged fields, s floats from one cell of the line to
// the next; at: 0 at the line's first cell, 1 at its last one, 2 between.
__device__ __forceinline__ float4 end_products(const float *su, const float *sd, const float *sl, int b, int s, int at,
                                               float dt, float rdx) {
    auto d1 = [&](const float *f) {
        if (at == 0) return g_head(f[b], f[b + s], f[b + 2 * s], f[b + 3 * s]) * rdx;
        if (at == 1) return g_tail(f[b - 3 * s], f[b - 2 * s], f[b - s], f[b]) * rdx;
        return g_central(f[b - 2 * s], f[b - s], f[b + s], f[b + 2 * s]) * rdx;
    };
    const float mu = dt * sl[b], dq = d1(sd), uq = d1(su);
    return make_float4(sd[b] * mu, dq * mu, su[b], mu * uq);
}

// The four terms of a cell `pp` from its line's end, from the products of the ten cells there (`stride` apart), as
// axis_edge sums them.
__device__ __forceinline__ float4 end_sums(const float4 *L, int stride, const float4 *taps, int pp, float sgn,
                                           float rdx) {
    float AT = 0.f, BT = 0.f, d2 = 0.f, g = 0.f;
#pragma unroll
    for (int r = 0; r < LEND; ++r) {
        const float4 l = L[r * stride], c = taps[r * ADJ_BAND + pp];
        AT = fmaf(c.x, l.x, AT);
        BT = fmaf(c.y, l.y, BT);
        d2 = fmaf(c.z, l.z, d2);
        g = fmaf(c.y, l.w, g);
    }
    return make_float4(AT * (rdx * rdx), sgn * BT * rdx, d2 * (rdx * rdx), sgn * g * rdx);
}

// Constants of the packed operations, each twice (in the constant bank).  (No packed product goes into a packed
// addition: see fk_pack.cuh.)
struct LineConsts {
    float2 c_1_12, c_m2_3, c_2_3, c_m1_12, rdx, neg_rdx, dt;
};
__device__ __forceinline__ float2 pair_central(const LineConsts &k, float2 m2, float2 m1, float2 p1, float2 p2) {
    return p_fma(k.c_m1_12, p2, p_fma(k.c_2_3, p1, p_fma(k.c_m2_3, m1, p_mul(k.c_1_12, m2))));
}
__device__ __forceinline__ Quad quad_central(const LineConsts &k, const Quad &m2, const Quad &m1, const Quad &p1,
                                             const Quad &p2) {
    return Quad{pair_central(k, m2.lo, m1.lo, p1.lo, p2.lo), pair_central(k, m2.hi, m1.hi, p1.hi, p2.hi)};
}
__device__ __forceinline__ Quad q_mul(const Quad &a, const Quad &b) {
    return Quad{p_mul(a.lo, b.lo), p_mul(a.hi, b.hi)};
}

// The x direction (along the four columns of a quad) at R cells that are at least ADJ_BAND from the columns' ends
// (others get values nobody reads), in two halves so that few values are live at a time.  of(f, t) is the cell
// t - 4 from the first one of field f (0: u, 1: D, 2: lambda_u).
//
// d2: u''; g: B^T (mu u').
template <int R, class Of>
__device__ __forceinline__ void cols_gd(const LineConsts &kc, Of of, Quad (&d2)[R], Quad (&g)[R]) {
    Quad U[R + 8], ux[R + 4], m[R + 4];
#pragma unroll
    for (int t = 0; t < 4; ++t) U[t] = of(0, t);
#pragma unroll
    for (int t = 0; t < R + 4; ++t) {
        U[t + 4] = of(0, t + 4);
        ux[t] = q_scale(quad_central(kc, U[t], U[t + 1], U[t + 3], U[t + 4]), kc.rdx);
        m[t] = q_mul(q_scale(of(2, t + 2), kc.dt), ux[t]);
    }
#pragma unroll
    for (int k = 0; k < R; ++k) {
        d2[k] = q_scale(quad_central(kc, ux[k], ux[k + 1], ux[k + 3], ux[k + 4]), kc.rdx);
        g[k] = q_scale(quad_central(kc, m[k], m[k + 1], m[k + 3], m[k + 4]), kc.neg_rdx);
    }
}

// at: A^T (D mu); bt: B^T ((B D) mu).
template <int R, class Of>
__device__ __forceinline__ void cols_at(const LineConsts &kc, Of of, Quad (&at)[R], Quad (&bt)[R]) {
    Quad D[R + 8], M[R + 8], q[R + 8], qx[R + 4], bx[R + 4];
    auto take = [&](int t) {
        D[t] = of(1, t);
        M[t] = q_scale(of(2, t), kc.dt);
        q[t] = q_mul(D[t], M[t]);
    };
#pragma unroll
    for (int t = 0; t < 4; ++t) take(t);
#pragma unroll
    for (int t = 0; t < R + 4; ++t) {
        take(t + 4);
        qx[t] = q_scale(quad_central(kc, q[t], q[t + 1], q[t + 3], q[t + 4]), kc.rdx);
        bx[t] = q_mul(q_scale(quad_central(kc, D[t], D[t + 1], D[t + 3], D[t + 4]), kc.rdx), M[t + 2]);
    }
#pragma unroll
    for (int k = 0; k < R; ++k) {
        at[k] = q_scale(quad_central(kc, qx[k], qx[k + 1], qx[k + 3], qx[k + 4]), kc.rdx);
        bt[k] = q_scale(quad_central(kc, bx[k], bx[k + 1], bx[k + 3], bx[k + 4]), kc.neg_rdx);
    }
}

// The same of the y direction, at the four cells 4 .. 7 of twelve along a row.  Results of a row lie in aligned
// pairs of registers: the outer taps as packed operations, the inner ones as scalar ones (see pg_central_row).
template <int N>
__device__ __forceinline__ void row_central(const LineConsts &k, const float (&a)[N + 4], float2 c, float (&d)[N]) {
#pragma unroll
    for (int t = 0; t < N; t += 2) {
        float2 s = p_mul(k.c_1_12, mk2(a[t], a[t + 1]));
        s.x = fmaf(-C_2_3, a[t + 1], s.x);
        s.y = fmaf(-C_2_3, a[t + 2], s.y);
        s.x = fmaf(C_2_3, a[t + 3], s.x);
        s.y = fmaf(C_2_3, a[t + 4], s.y);
        s = p_mul(p_fma(k.c_m1_12, mk2(a[t + 4], a[t + 5]), s), c);
        d[t] = s.x;
        d[t + 1] = s.y;
    }
}
template <int N, int M>
__device__ __forceinline__ void row_mul(const float (&a)[M], const float (&b)[N], float (&d)[N]) {
    constexpr int off = (M - N) / 2;
#pragma unroll
    for (int t = 0; t < N; t += 2) {
        const float2 s = p_mul(mk2(a[t + off], a[t + off + 1]), mk2(b[t], b[t + 1]));
        d[t] = s.x;
        d[t + 1] = s.y;
    }
}
__device__ __forceinline__ void row_gd(const LineConsts &kc, const float (&U)[12], const float (&mu)[12],
                                       float (&d2)[4], float (&g)[4]) {
    float uy[8], m[8];
    row_central<8>(kc, U, kc.rdx, uy);
    row_mul<8, 12>(mu, uy, m);
    row_central<4>(kc, uy, kc.rdx, d2);
    row_central<4>(kc, m, kc.neg_rdx, g);
}
__device__ __forceinline__ void row_at(const LineConsts &kc, const float (&D)[12], const float (&mu)[12],
                                       float (&at)[4], float (&bt)[4]) {
    float q[12], qy[8], by[8];
    row_mul<12, 12>(D, mu, q);
    row_central<8>(kc, q, kc.rdx, qy);
    row_central<8>(kc, D, kc.rdx, by);
    row_mul<8, 12>(mu, by, by);
    row_central<4>(kc, qy, kc.rdx, at);
    row_central<4>(kc, by, kc.neg_rdx, bt);
}

// Sums 16 values over a warp: lane i < 16 returns the sum of v[i] (lanes 16..31 the same).  Each
// exchange halves the values a lane still carries: 16 exchanges instead of 5 per value.
__device__ __forceinline__ float warp_sum16(float (&v)[16]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int h = 8; h >= 1; h >>= 1) {
        const bool up = (lane & h) != 0;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            if (k >= h) break;
            const float keep = up ? v[k + h] : v[k], give = up ? v[k] : v[k + h];
            v[k] = keep + __shfl_xor_sync(0xffffffffu, give, h);
        }
    }
    return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 16);
}

__device__ __forceinline__ void cp_async16(float *dst, const float *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}

// The tiles of a launch: block (x, y, e) takes tile (x, y) of a cut of the grid (rows in groups of LR,
// columns in quads, dealt out evenly, the larger shares last) of experiment e.  No division is left to the
// device: a thread has a few cells, and one division costs as much as one of them.
struct LineRun {
    int64_t state, lam, plane, theta;  // elements from one experiment to the next: state, cotangent, gD, gtheta
    const AdjointArgs *exps;           // the experiments' stimuli; null: one experiment, those of the arguments
    int early;                         // the launch before is the reverse step before, or waits for it
    int g_each, g_small, q_each, q_small;  // groups (quads) of a tile, and tiles that have one less
    int inv[2], inv_q[2];                  // 2^16 / groups of a tile (/ its quads + 2), rounded up: for the
                                           // tiles that have one less, and for the others
    LineConsts kc;
};

// The arguments stay in the constant bank, for many experiments those of the first one and the distance to
// the others.  With programmatic dependent launch the state and D, which no reverse step writes, are fetched
// before the step before has ended.  (Measured with the regrouped operators, us per step: arguments copied from
// memory and all loads after the step before 28.4 for 16 experiments of 256^2, 7.1 for 151 x 203, against 24.2 and
// 5.0; blocks that walk over tiles, the next one's loads in flight, 28.1: their shares are fixed, some take four
// tiles where 3.4 are the mean; three blocks per SM, at 80 registers, spill: 24.0, but 512^2 9.5 against 7.4.)
//
// SHARE: threads that share a unit.  What a thread does once per tile (places, addresses, loads, sums) costs
// it as much as two cells, so many tiles take two threads per unit (tiles of 16 x 64 cells); where all tiles
// run at once the chain of a thread counts, and four take it (16 x 32).  us per step with 2 | 4: 151 x 203
// 6.3 | 5.0, 16 of 64^2 6.9 | 5.2, 4 of 100 x 400 7.9 | 9.0, 512^2 (512 tiles of 16 x 32 on 304 places) 7.9 | 9.7,
// 16 of 256^2 24.8 | 29.0.
template <int SHARE>
__global__ void __launch_bounds__(LNT, 2)
    fk_adjoint_line_kernel(const __grid_constant__ AdjointArgs a, const __grid_constant__ LineRun b) {
    using T_ = LineTile<SHARE>;
    constexpr int LU = T_::LU, LSW = T_::LSW, LSH = T_::LSH;
    constexpr int LC = T_::LC;
    // u, D and lambda_u with 4 cells around; a unit's own v, w, lambda_v, lambda_w, the first then its lambda_u
    // through the currents; the x direction's A^T, B^T, u'', B^T (mu u'); the products at the
    // ends of the columns ([r][column]) and of the rows ([end][r][row]), the four terms of the rows' bands
    // ([end][pp][row]) and the corner tables
    extern __shared__ __align__(16) float line_smem[];
    float *const su = line_smem, *const sd = su + LSH * LSW, *const sl = sd + LSH * LSW;
    float4(*const sp)[LR][LU] = reinterpret_cast<float4(*)[LR][LU]>(sl + LSH * LSW);
    float4(*const sr)[LR][LU] = sp + 4;
    float4 *const ex = reinterpret_cast<float4 *>(sr + 4);
    float4 *const ey = ex + LEND * LC, *const yr = ey + 2 * LEND * LROWS, *const taps = yr + 2 * ADJ_BAND * LROWS;
    constexpr int PT_WARPS = SHARE == 4 ? 2 * LU / 32 : LU / 32;
    __shared__ float red[PT_WARPS][16];
    const int tid = threadIdx.x, lane = tid & 31;
    const int role = tid / LU, unit = tid % LU;
    const int H = a.H, W = a.W, pitch = a.pitch;
    const float dt = a.dt, rdx = a.rdx;

    const int bx = blockIdx.x, by = blockIdx.y;
    const int64_t e = blockIdx.z;
    const int G = b.g_each - (by < b.g_small), tq = b.q_each - (bx < b.q_small);  // groups and quads
    // the last tile row's groups are aligned to the bottom, so that rows 0 and H-1 are the first and the last
    // row of a thread; rows above the tile's own belong to the tile above
    const int shift = by == (int)gridDim.y - 1 ? H & (LR - 1) : 0;
    const int row0 = (by * b.g_each - min(by, b.g_small)) * LR - shift;  // the first group's first row
    const int j0 = 4 * (bx * b.q_each - min(bx, b.q_small));
    // units by pairs of quad columns: those near the left and right sides then lie in few warps
    const int pair = (unit >> 1) * b.inv[by >= b.g_small] >> 16;
    const bool mine = 2 * pair + (unit & 1) < tq;
    const int lq = mine ? 2 * pair + (unit & 1) : 0, lg = mine ? (unit >> 1) - pair * G : 0;
    const int i0 = row0 + lg * LR, j = j0 + 4 * lq;
    const int k_lo = lg == 0 ? shift : 0;  // rows before it belong to the tile above
    const int64_t off0 = (int64_t)i0 * pitch + j;
    const int64_t e_state = e * b.state, e_lam = e * b.lam, e_plane = e * b.plane;

    // the staged quads that this thread brings in: f(row, quad)
    auto each_quad = [&](auto f) {
        const int per = tq + 2, n = (G * LR + 8) * per, inv = b.inv_q[bx >= b.q_small];
#pragma unroll
        for (int pass = 0; pass < ((LG * LR + 8) * (T_::LQ + 2) + LNT - 1) / LNT; ++pass) {
            const int x = tid + pass * LNT, r = x * inv >> 16;
            if (x < n) f(r, x - r * per);
        }
    };
    // Starts the loads of the state and D, or of the cotangent (all through L2: with programmatic dependent
    // launch L1 may hold lines of the step before the last).
    auto load = [&](bool state, bool lam) {
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        each_quad([&](int r, int q) {
            const int i = row0 - 4 + r, jc = j0 - 4 + 4 * q, o = r * LSW + 4 * q;
            const bool col_in = jc >= 0 && jc < W;  // (the quads outside: below)
            const int64_t g = (int64_t)clampi(i, 0, H - 1) * pitch + jc;
            if (state && col_in) {
                cp_async16(su + o, a.u + e_state + g);
                cp_async16(sd + o, a.D + g);
            }
            if (lam) {
                if (col_in && i >= 0 && i < H) cp_async16(sl + o, a.lu + e_lam + g);
                else *reinterpret_cast<float4 *>(sl + o) = zero;
            }
        });
        // a unit's v, w, lambda_v, lambda_w, dealt out over its threads
#pragma unroll
        for (int x = 0; x < 4 / SHARE; ++x) {
            const int f = role + SHARE * x;
            if (!(f < 2 ? state : lam)) continue;
            const float *const src = (f == 0 ? a.v : f == 1 ? a.w : f == 2 ? a.lv : a.lw) + (f < 2 ? e_state : e_lam) + off0;
#pragma unroll
            for (int k = 0; k < LR; ++k) {
                if (mine && k >= k_lo) cp_async16(reinterpret_cast<float *>(&sp[f][k][unit]), src + (int64_t)k * pitch);
                else sp[f][k][unit] = zero;
            }
        }
    };
    if (b.early) load(true, false);
    const bool left = bx == 0, right = bx == (int)gridDim.x - 1, top = by == 0, bottom = by == (int)gridDim.y - 1;
    if (left || right || top || bottom)
        for (int x = tid; x < LEND * ADJ_BAND; x += LNT)
            taps[x] = __ldg(reinterpret_cast<const float4 *>(&kEndTaps) + x);
    grid_dependency_wait();
    grid_launch_dependents();
    load(!b.early, true);

    double *const slot = a.gtheta + e * b.theta + (int64_t)(by * (int)gridDim.x + bx) * kAdjParamStride + (tid < 12 ? tid : 0);
    const double slot_was = a.gtheta && tid < 12 ? __ldcg(slot) : 0.0;  // early: its trip overlaps the work
    const Stim *const stims = b.exps ? b.exps[e].stim : a.stim;
    unsigned active = 0;
    if (role < SHARE / 2) {
        const int n_stim = b.exps ? b.exps[e].n_stim : a.n_stim;
        active = __ballot_sync(0xffffffffu, lane < n_stim && stim_active(stims[lane < kMaxStim ? lane : 0], a.t));
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    // A thread's own loads have arrived: at the grid's left and right sides the nearest cell takes the place
    // of those of u and D outside, zero that of lambda.
    if (left || right) {
        const int n = W - 1 - (j0 + 4 * (tq - 1));  // the last cell's place in the last quad
        each_quad([&](int r, int c) {
            const bool first = left && c == 1, last = right && c == tq;
            if (!first && !last) return;
#pragma unroll
            for (int f = 0; f < 3; ++f) {
                float4 *const q = reinterpret_cast<float4 *>(line_smem + f * LSH * LSW + r * LSW) + c;
                float4 y = *q;
                if (f < 2 && first) q[-1] = make_float4(y.x, y.x, y.x, y.x);
                if (last) {
                    if (n < 1) y.y = f < 2 ? y.x : 0.0f;
                    if (n < 2) y.z = f < 2 ? y.y : 0.0f;
                    if (n < 3) y.w = f < 2 ? y.z : 0.0f;
                    q[0] = y;
                    if (f < 2) q[1] = make_float4(y.w, y.w, y.w, y.w);
                }
            }
        });
    }
    __syncthreads();

    // ---- the bands: products at the ends of the tile's lines, then the sums of the cells there ------------
    if (left || right || top || bottom) {
        const int rows = G * LR, first = 4 * LSW + 4;  // the tile's rows; its first cell's place
        if (top || bottom)
            for (int x = tid; x < LEND * LC; x += LNT) {
                const int r = x / LC, c = x % LC;
                if (c < 4 * tq)
                    ex[x] = end_products(su, sd, sl, first + (top ? r : rows - 1 - r) * LSW + c, LSW,
                                         r > 0 ? 2 : top ? 0 : 1, dt, rdx);
            }
        for (int x = tid; x < 2 * LEND * LROWS; x += LNT) {
            const int end = x / (LEND * LROWS), r = x / LROWS % LEND, row = x % LROWS;
            if (row < rows && (end ? right : left))
                ey[x] = end_products(su, sd, sl, first + row * LSW + (end ? W - 1 - j0 - r : r), 1, r > 0 ? 2 : end, dt,
                                     rdx);
        }
        __syncthreads();
        if (top || bottom)
            for (int x = tid; x < ADJ_BAND * LC; x += LNT) {
                const int pp = x / LC, c = x % LC;
                if (c >= 4 * tq) continue;
                const float4 y = end_sums(ex + c, LC, taps, pp, top ? 1.0f : -1.0f, rdx);
                // the cell's unit (see `pair`), its row there and its place in the quad
                const int row = top ? pp : rows - 1 - pp, q = c >> 2;
                const int un = 2 * ((q >> 1) * G + (row >> 1)) + (q & 1);
                float *const to = reinterpret_cast<float *>(&sr[0][row & 1][un]) + (c & 3);
                constexpr int plane = 4 * LR * LU;
                to[0] = y.x;
                to[plane] = y.y;
                to[2 * plane] = y.z;
                to[3 * plane] = y.w;
            }
        for (int x = tid; x < 2 * ADJ_BAND * LROWS; x += LNT) {
            const int end = x / (ADJ_BAND * LROWS), pp = x / LROWS % ADJ_BAND, row = x % LROWS;
            if (row < rows && (end ? right : left))
                yr[x] = end_sums(ey + end * LEND * LROWS + row, LROWS, taps, pp, end ? -1.0f : 1.0f, rdx);
        }
    }

    // Four threads of a unit: 0 and 1 take the pointwise part of its two rows, 2 and 3 the two halves of the
    // x direction (along rows); then each one half of the y direction of one of the rows.  Two
    // threads: 0 the pointwise part, 1 the x direction; then each the y direction of one row.
    const int base = (lg * LR + 4) * LSW + 4 * lq + 4;  // the unit's first cell
    if (role < SHARE / 2) {
        const Model &md = a.m;
        float gth[16];
#pragma unroll
        for (int q = 0; q < 16; ++q) gth[q] = 0.0f;
#pragma unroll 1
        for (int k = SHARE == 4 ? role : 0; k < (SHARE == 4 ? role + 1 : LR); ++k) {
            const bool stored = mine && k >= k_lo;
            const int64_t o = off0 + (int64_t)k * pitch;
            float4 v4 = sp[0][k][unit], w4 = sp[1][k][unit];
            float4 lv4 = sp[2][k][unit], lw4 = sp[3][k][unit];
            const float4 u4 = *reinterpret_cast<const float4 *>(su + base + k * LSW);
            const float4 l4 = *reinterpret_cast<const float4 *>(sl + base + k * LSW);
            const int i = i0 + k;
            if (j + 3 >= W) {  // columns beyond W: whatever lies in the padding (lambda_u is zero there)
                if (j + 1 >= W) v4.y = w4.y = lv4.y = lw4.y = 0.f;
                if (j + 2 >= W) v4.z = w4.z = lv4.z = lw4.z = 0.f;
                if (j + 3 >= W) v4.w = w4.w = lv4.w = lw4.w = 0.f;
            }
            unsigned replaced = 0;  // cells whose current a stimulus replaces
            if (active && stored)
                for (unsigned x = active; x; x &= x - 1) {
                    const Stim &st = stims[__ffs(x) - 1];
                    float4 f;
                    if (st.field) {
                        f = __ldg(reinterpret_cast<const float4 *>(st.field + o));
                    } else {
                        const bool in = i >= st.r0 && i < st.r1;
                        f.x = in && j >= st.c0 && j < st.c1 ? st.amplitude : 0.0f;
                        f.y = in && j + 1 >= st.c0 && j + 1 < st.c1 ? st.amplitude : 0.0f;
                        f.z = in && j + 2 >= st.c0 && j + 2 < st.c1 ? st.amplitude : 0.0f;
                        f.w = in && j + 3 >= st.c0 && j + 3 < st.c1 ? st.amplitude : 0.0f;
                    }
                    replaced |= (f.x != 0.0f ? 1u : 0u) | (f.y != 0.0f ? 2u : 0u) | (f.z != 0.0f ? 4u : 0u) |
                                (f.w != 0.0f ? 8u : 0u);
                }
            const float uu[4] = {u4.x, u4.y, u4.z, u4.w}, ll[4] = {l4.x, l4.y, l4.z, l4.w};
            const float vv[4] = {v4.x, v4.y, v4.z, v4.w}, ww[4] = {w4.x, w4.y, w4.z, w4.w};
            const float lvv[4] = {lv4.x, lv4.y, lv4.z, lv4.w}, lww[4] = {lw4.x, lw4.y, lw4.z, lw4.w};
            float ov[4], ow[4], pu[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const float u = uu[c], v = vv[c], w = ww[c], lv = lvv[c], lw = lww[c], lu = ll[c];
                const bool stim = (replaced >> c & 1u) != 0;
                const bool p = u >= md.V_c, q = u >= md.V_v;
                const float uk = u - md.V_csi;
                const float S = one_plus_tanh(md.k * uk);  // 1 + tanh
                const float sech2 = S * (2.0f - S);        // 1 - tanh^2
                const float uc = u - md.V_c, u1 = 1.0f - u;
                // the cotangents: adjoint_pointwise's operations
                const float mu = dt * lu;
                const float dvdv = 1.0f + dt * (p ? -md.r_tau_vp : -(q ? md.r_tau_v2m : md.r_tau_v1m));
                const float dwdw = 1.0f + dt * (p ? -md.r_tau_wp : -md.r_tau_wm);
                const float dfi = p ? -v * (1.0f + md.V_c - 2.0f * u) * md.r_tau_d : 0.0f;
                const float dso = p ? 0.0f : md.r_tau_0;
                const float dsi = -w * md.k * sech2 * md.r_2tau_si;
                const float dJdu = stim ? 0.0f : -(dfi + dso + dsi) * md.r_Cm;
                const float dJdv = stim || !p ? 0.0f : uc * u1 * md.r_tau_d * md.r_Cm;
                const float dJdw = stim ? 0.0f : S * md.r_2tau_si * md.r_Cm;
                ov[c] = lv * dvdv + mu * dJdv;
                ow[c] = lw * dwdw + mu * dJdw;
                pu[c] = lu * (1.0f + dt * dJdu);
                const float lj = stim || !stored ? 0.0f : lu;  // lambda_u where the current is the model's
                // parameter sums without their constant factors (cardiax/params.py fields 0..11)
                const float lvp = p ? lv : 0.0f, lvo = (lv - lvp) * (1.0f - v), lvq = q ? lvo : 0.0f;
                const float lwp = p ? lw : 0.0f;
                gth[0] = fmaf(lvp, v, gth[0]);
                gth[1] += lvo - lvq;
                gth[2] += lvq;
                gth[3] = fmaf(lwp, w, gth[3]);
                gth[4] = fmaf(lw - lwp, 1.0f - w, gth[4]);
                const float jp = p ? lj : 0.0f, jv = jp * v * u1, jw = lj * w, js = jw * sech2;
                gth[5] = fmaf(jv, uc, gth[5]);
                gth[6] = fmaf(lj - jp, u, gth[6]);
                gth[7] += jp;
                gth[8] = fmaf(jw, S, gth[8]);
                gth[9] = fmaf(js, uk, gth[9]);
                gth[10] += js;
                gth[11] += jv;
            }
            sp[0][k][unit] = make_float4(pu[0], pu[1], pu[2], pu[3]);
            if (stored) {
                if (j + 3 < W) {
                    *reinterpret_cast<float4 *>(a.olv + e_lam + o) = make_float4(ov[0], ov[1], ov[2], ov[3]);
                    *reinterpret_cast<float4 *>(a.olw + e_lam + o) = make_float4(ow[0], ow[1], ow[2], ow[3]);
                } else {
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        if (j + c < W) {
                            a.olv[e_lam + o + c] = ov[c];
                            a.olw[e_lam + o + c] = ow[c];
                        }
                }
            }
        }
        if (a.gtheta) {
            const float x = warp_sum16(gth);
            if (lane < 16) red[tid / 32][lane] = x;
        }
    } else {
        Quad x[LR], y[LR];
        auto of = [&](int f, int t) { return ld_quad((f == 0 ? su : f == 1 ? sd : sl) + base + (t - 4) * LSW); };
        // (units in the band have their sums already)
        const bool band = mine && (i0 < ADJ_BAND || i0 >= H - ADJ_BAND);
        auto keep = [&](int f, Quad (&z)[LR]) {
#pragma unroll
            for (int k = 0; k < LR; ++k)
                if (!band) sr[f][k][unit] = make_float4(z[k].lo.x, z[k].lo.y, z[k].hi.x, z[k].hi.y);
        };
        if (SHARE == 2 || role == 2) {
            cols_gd<LR>(b.kc, of, x, y);
            keep(2, x);
            keep(3, y);
        }
        if (SHARE == 2 || role == 3) {
            cols_at<LR>(b.kc, of, x, y);
            keep(0, x);
            keep(1, y);
        }
    }
    const int k = role & 1;
    const bool stored = mine && k >= k_lo;
    const bool takes_gd = SHARE == 2 || role < 2, takes_at = SHARE == 2 || role >= 2;
    const int64_t o = off0 + (int64_t)k * pitch;
    float4 gd4 = make_float4(0.f, 0.f, 0.f, 0.f);
    if (takes_gd && a.gD && stored) gd4 = __ldcg(reinterpret_cast<const float4 *>(a.gD + e_plane + o));
    float yt[4][4], mu[4];  // A^T, B^T, u'' and B^T (mu u') of the y direction
    {
        const int c0 = base + k * LSW;
        float M[12], F[12];
        auto row = [&](const float *p, float (&x)[12]) {
#pragma unroll
            for (int t = 0; t < 3; ++t) {
                const float4 q = *reinterpret_cast<const float4 *>(p + c0 + 4 * t - 4);
                x[4 * t] = q.x, x[4 * t + 1] = q.y, x[4 * t + 2] = q.z, x[4 * t + 3] = q.w;
            }
        };
        row(sl, M);
#pragma unroll
        for (int t = 0; t < 12; t += 2) {
            const float2 x = p_mul(mk2(M[t], M[t + 1]), b.kc.dt);
            M[t] = x.x, M[t + 1] = x.y;
        }
        row(takes_gd ? su : sd, F);
        if (takes_gd) row_gd(b.kc, F, M, yt[2], yt[3]);
        if (takes_at) {
            if (takes_gd) row(sd, F);
            row_at(b.kc, F, M, yt[0], yt[1]);
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) mu[c] = M[c + 4];
    }
    __syncthreads();
    // the row's cells in a band
    if ((left && j < ADJ_BAND) || (right && j + 3 >= W - ADJ_BAND)) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int far = W - 1 - j - c;
            const bool near0 = left && j + c < ADJ_BAND;
            if (!near0 && !(right && far >= 0 && far < ADJ_BAND)) continue;
            const float4 y = yr[((near0 ? 0 : ADJ_BAND) + (near0 ? j + c : far)) * LROWS + lg * LR + k];
            yt[0][c] = y.x;
            yt[1][c] = y.y;
            yt[2][c] = y.z;
            yt[3][c] = y.w;
        }
    }
    auto put = [&](const float (&z)[4], float *out) {
        if (j + 3 < W) {
            __stcg(reinterpret_cast<float4 *>(out), make_float4(z[0], z[1], z[2], z[3]));
        } else {
#pragma unroll
            for (int c = 0; c < 4; ++c)
                if (j + c < W) __stcg(out + c, z[c]);
        }
    };
    auto four = [](float4 q, float (&x)[4]) { x[0] = q.x, x[1] = q.y, x[2] = q.z, x[3] = q.w; };
    float z[4], x0[4], x1[4];
    if (stored && takes_at) {
        four(sp[0][k][unit], z);
        four(sr[0][k][unit], x0);
        four(sr[1][k][unit], x1);
#pragma unroll
        for (int c = 0; c < 4; ++c) z[c] = z[c] + ((x0[c] + yt[0][c]) + (x1[c] + yt[1][c]));
        put(z, a.olu + e_lam + o);
    }
    if (stored && takes_gd && a.gD) {
        four(gd4, z);
        four(sr[2][k][unit], x0);
        four(sr[3][k][unit], x1);
#pragma unroll
        for (int c = 0; c < 4; ++c) z[c] = z[c] + (mu[c] * (x0[c] + yt[2][c]) + (x1[c] + yt[3][c]));
        put(z, a.gD + e_plane + o);
    }
    if (a.gtheta && tid < 12) {
        double x = 0.0;
#pragma unroll
        for (int w = 0; w < PT_WARPS; ++w) x += (double)red[w][tid];
        __stcg(slot, fma(a.theta_factor[tid], x, slot_was));
    }
}

// The device copy of an experiment's arguments, moved to step k of its segment (see
// fk_adjoint_batch_kernel); all threads, two barriers.
__device__ __forceinline__ void stage_experiment(AdjointArgs &sa, const AdjointArgs *exps, int64_t k_stride,
                                                 int k, int parity, float t) {
    const uint32_t *src = reinterpret_cast<const uint32_t *>(exps + blockIdx.z);
    uint32_t *dst = reinterpret_cast<uint32_t *>(&sa);
    for (int w = threadIdx.x; w < (int)(sizeof(AdjointArgs) / 4); w += blockDim.x) dst[w] = __ldg(src + w);
    __syncthreads();
    if (threadIdx.x == 0) {
        const int64_t o = (int64_t)k * k_stride;
        sa.u += o;
        sa.v += o;
        sa.w += o;
        sa.t = t;
        if (parity) {
            const float *lu = sa.lu, *lv = sa.lv, *lw = sa.lw;
            sa.lu = sa.olu;
            sa.lv = sa.olv;
            sa.lw = sa.olw;
            sa.olu = const_cast<float *>(lu);
            sa.olv = const_cast<float *>(lv);
            sa.olw = const_cast<float *>(lw);
        }
    }
    __syncthreads();
}

// One reverse step of many experiments (blockIdx.z): exps[e] describes step 0 of experiment e's
// segment with the cotangent ping-pong buffers (lu.. = buffer A, olu.. = buffer B); step k reads
// the state k * k_stride further on, and parity 1 swaps the two cotangent buffers.
__global__ void __launch_bounds__(ANT, 4) fk_adjoint_batch_kernel(const AdjointArgs *__restrict__ exps,
                                                               int64_t k_stride, int k, int parity,
                                                               float t) {
    __shared__ __align__(16) AdjointArgs sa;
    stage_experiment(sa, exps, k_stride, k, parity, t);
    adjoint_tile(sa, blockIdx.x, blockIdx.y, gridDim.x);
}

// Sums over the experiments in their order: dL/dD to the dense H x W plane oD, and (the last block) dL/dtheta,
// over the slots as well, to oth.
__global__ void __launch_bounds__(32 * kAdjParams)
    fk_adjoint_sum_kernel(const float *gD, const double *gtheta, int n_exp, int H, int W, int pitch, int slots,
                          float *oD, float *oth) {
    if (blockIdx.x == gridDim.x - 1) {
        const int p = threadIdx.x / 32, lane = threadIdx.x % 32;
        double sum = 0.0;
        for (int e = 0; e < n_exp; ++e) {
            double x = 0.0;
            for (int k = lane; k < slots; k += 32) x += __ldg(gtheta + ((int64_t)e * slots + k) * kAdjParamStride + p);
            for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
            sum += x;
        }
        if (lane == 0) oth[p] = (float)sum;
        return;
    }
    const int64_t plane = (int64_t)H * pitch, quads = (int64_t)H * (pitch / 4);
    for (int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; x < quads;
         x += (int64_t)(gridDim.x - 1) * blockDim.x) {
        const int i = (int)(x / (pitch / 4)), j = 4 * (int)(x - (int64_t)i * (pitch / 4));
        if (j >= W) continue;
        const float *src = gD + (int64_t)i * pitch + j;
        float4 s = __ldg(reinterpret_cast<const float4 *>(src));
#pragma unroll 8
        for (int e = 1; e < n_exp; ++e) {
            const float4 y = __ldg(reinterpret_cast<const float4 *>(src + e * plane));
            s = make_float4(s.x + y.x, s.y + y.y, s.z + y.z, s.w + y.w);
        }
        float *out = oD + (int64_t)i * W + j;
        const float f[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
        for (int m = 0; m < 4; ++m)
            if (j + m < W) out[m] = f[m];
    }
}

// Which kernel takes a grid, and its blocks.
bool long_lines(int H, int W) { return H >= kLineMin && W >= kLineMin; }
dim3 adjoint_grid(int H, int W, int n_exp) {
    return dim3((W + ATX - 1) / ATX, (H + ATY - 1) / ATY, n_exp);
}
template <int SHARE>
dim3 line_grid(int H, int W) {
    constexpr int LQ = LineTile<SHARE>::LQ;
    return dim3(((W + 3) / 4 + LQ - 1) / LQ, ((H + LR - 1) / LR + LG - 1) / LG);
}

template <int SHARE>
cudaError_t launch_line_as(const AdjointArgs &a, LineRun b, int n_exp, cudaStream_t stream) {
    const dim3 cut = line_grid<SHARE>(a.H, a.W);
    const int ng = (a.H + LR - 1) / LR, nq = (a.W + 3) / 4, nbx = (int)cut.x, nby = (int)cut.y;
    b.g_each = (ng + nby - 1) / nby;
    b.g_small = b.g_each * nby - ng;
    b.q_each = (nq + nbx - 1) / nbx;
    b.q_small = b.q_each * nbx - nq;
    for (int q = 0; q < 2; ++q) {  // (shares of five groups, or three quads, at least)
        b.inv[q] = (65536 + b.g_each - 2 + q) / (b.g_each - 1 + q);
        b.inv_q[q] = (65536 + b.q_each + q) / (b.q_each + 1 + q);
    }
    auto twice = [](float x) { return float2{x, x}; };
    b.kc = LineConsts{twice(C_1_12), twice(-C_2_3), twice(C_2_3), twice(-C_1_12), twice(a.rdx), twice(-a.rdx),
                      twice(a.dt)};
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(nbx, nby, n_exp);
    cfg.blockDim = dim3(LNT);
    cfg.dynamicSmemBytes = LineTile<SHARE>::SMEM;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, fk_adjoint_line_kernel<SHARE>, a, b);
}

cudaError_t launch_line(const AdjointArgs &a, LineRun b, int n_exp, bool chained, cudaStream_t stream) {
    // the attribute is per function and per context: set again whenever the context changes
    static thread_local uint64_t configured_ctx = 0;
    static thread_local int n_sm = 0;
    if (context_changed(configured_ctx)) {
        cudaError_t e;
        int dev = -1;
        if ((e = cudaGetDevice(&dev)) != cudaSuccess ||
            (e = cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess ||
            (e = cudaFuncSetAttribute(fk_adjoint_line_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      LineTile<2>::SMEM)) != cudaSuccess ||
            (e = cudaFuncSetAttribute(fk_adjoint_line_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      LineTile<4>::SMEM)) != cudaSuccess) {
            configured_ctx = 0;
            return e;
        }
    }
    b.early = chained;
    const dim3 cut = line_grid<4>(a.H, a.W);
    const bool at_once = (int64_t)cut.x * cut.y * n_exp <= 2 * n_sm;
    return at_once ? launch_line_as<4>(a, b, n_exp, stream) : launch_line_as<2>(a, b, n_exp, stream);
}

}  // namespace

void set_theta_factors(AdjointArgs &a) {
    const Model &m = a.m;
    const double d = a.dt, cm = m.r_Cm, si = m.r_2tau_si;
    const double f[12] = {
        d * m.r_tau_vp * m.r_tau_vp,      // tau_v_plus
        -d * m.r_tau_v1m * m.r_tau_v1m,   // tau_v1_minus
        -d * m.r_tau_v2m * m.r_tau_v2m,   // tau_v2_minus
        d * m.r_tau_wp * m.r_tau_wp,      // tau_w_plus
        -d * m.r_tau_wm * m.r_tau_wm,     // tau_w_minus
        -d * m.r_tau_d * m.r_tau_d * cm,  // tau_d
        d * m.r_tau_0 * m.r_tau_0 * cm,   // tau_0
        d * m.inv_tau_r * m.inv_tau_r * cm,  // tau_r
        -d * 2.0 * si * si * cm,          // tau_si
        d * si * cm,                      // k
        -d * m.k * si * cm,               // V_csi
        -d * m.r_tau_d * cm,              // V_c
    };
    for (int k = 0; k < 12; ++k) a.theta_factor[k] = f[k];
}

int64_t adjoint_slots(int H, int W) {
    const dim3 g = long_lines(H, W) ? line_grid<4>(H, W) : adjoint_grid(H, W, 1);
    return (int64_t)g.x * g.y;
}

cudaError_t launch_adjoint(const AdjointArgs &a, bool chained, cudaStream_t stream) {
    if (long_lines(a.H, a.W)) {
        return launch_line(a, LineRun{}, 1, chained, stream);
    }
    fk_adjoint_kernel<<<adjoint_grid(a.H, a.W, 1), ANT, 0, stream>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_adjoint_batch(const AdjointArgs &first, const AdjointArgs *exps, int n_exp, int64_t exp_stride,
                                 int k, int parity, float t, bool chained, cudaStream_t stream) {
    if (n_exp < 1) return cudaSuccess;
    const int64_t plane = (int64_t)first.H * first.pitch, ns = 3 * plane;
    if (!long_lines(first.H, first.W)) {
        fk_adjoint_batch_kernel<<<adjoint_grid(first.H, first.W, n_exp), ANT, 0, stream>>>(exps, ns, k, parity, t);
        return cudaGetLastError();
    }
    AdjointArgs a = first;
    a.u += k * ns;
    a.v += k * ns;
    a.w += k * ns;
    a.t = t;
    if (parity) {
        const float *const lu = a.lu, *const lv = a.lv, *const lw = a.lw;
        a.lu = a.olu;
        a.lv = a.olv;
        a.lw = a.olw;
        a.olu = const_cast<float *>(lu);
        a.olv = const_cast<float *>(lv);
        a.olw = const_cast<float *>(lw);
    }
    LineRun b{};
    b.exps = exps;
    b.state = exp_stride;
    b.lam = ns;
    b.plane = plane;
    b.theta = adjoint_slots(a.H, a.W) * kAdjParamStride;
    return launch_line(a, b, n_exp, chained, stream);
}

cudaError_t launch_adjoint_sum(const float *gD, const double *gtheta, int n_exp, int H, int W, int pitch, float *oD,
                               float *oth, cudaStream_t stream) {
    const int64_t quads = (int64_t)H * (pitch / 4), n = 32 * kAdjParams;
    const int64_t blocks = (quads + n - 1) / n;
    fk_adjoint_sum_kernel<<<(int)(blocks < 1024 ? blocks : 1024) + 1, (int)n, 0, stream>>>(
        gD, gtheta, n_exp, H, W, pitch, (int)adjoint_slots(H, W), oD, oth);
    return cudaGetLastError();
}

}  // namespace fk
