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
#include "fk_math.cuh"
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

// ---- lines of at least kLineMin cells: two threads per unit of two rows of a quad, one stage -------
// What bounds it: the tile kernel above stages six derivative planes, reads ten-cell products for
// each cell of the 6-cell edge band, tests every stimulus's protocol in every cell and reduces 13
// parameter sums over a warp for every two cells (us per step: 39.5 for 16 experiments of 256^2,
// 10.9 for one 151 x 203 grid, 10.5 for 16 of 64^2).  Here everything comes from one staged tile of
// u, D and lambda_u and stays in registers: 28.6, 7.1 and 7.9 us.  At 16 x 256^2 a step executes 400
// instructions per cell at 42 % of the issue slots; one small grid waits for its loads (0.5 us),
// then for the longest chain of a unit, 2500 cycles for each half of it.  The operations are fewer
// because they are regrouped:
//   * both transposed products of an axis share their second operator,
//       A^T (D mu) + B^T ((B D) mu) = (E^T G^T / dx) (G^T C^T (D mu) / dx + C^T (B D) mu),
//   * G^T on central rows is -G; the one-sided rows 0 and N-1 (and the pad rows -1 and N in the
//     second operator) are taken out of the central sum and added as rank-one terms to the four
//     cells they reach, only by the warps that hold such cells,
//   * 1/dx^2, dt and the constant factors of the parameter sums are applied once, to the sums, and a
//     parameter sum is reduced over a warp once per 8 cells.
constexpr int kLineMin = 20;  // shorter lines (fewer than three quads or nine rows in a last tile)
                              // take the tile kernel above
constexpr int LR = 2;         // rows per thread
constexpr int LG = 8, LQ = 16;                   // most row groups and quads of a tile
constexpr int LU = LG * LQ;                      // units of a tile; two threads share one
constexpr int LNT = 2 * LU;
constexpr int LSW = 4 * LQ + 12;                 // staged row: 4 cells on either side, and 4 more so
                                                 // that 8 lanes (2 quads of 4 groups) read from 8
                                                 // different 16-byte banks
constexpr int LSH = LG * LR + 8 + 1;             // 4 rows above and below; the first group of the
                                                 // last tile row may reach one row further up

__constant__ float kHeadC[4] = {C_HEAD0, C_THREE, -C_3_2, C_1_3};
__constant__ float kTailC[4] = {C_TAIL0, C_3_2, -C_THREE, C_TAIL3};

struct V4 {
    float x, y, z, w;
};
__device__ __forceinline__ V4 ld_v4(const float *p) {
    const float4 v = *reinterpret_cast<const float4 *>(p);
    return V4{v.x, v.y, v.z, v.w};
}
__device__ __forceinline__ V4 vmul(V4 a, V4 b) { return V4{a.x * b.x, a.y * b.y, a.z * b.z, a.w * b.w}; }
__device__ __forceinline__ V4 vscale(float c, V4 a) { return V4{c * a.x, c * a.y, c * a.z, c * a.w}; }
__device__ __forceinline__ V4 vfma(V4 a, V4 b, V4 c) {
    return V4{fmaf(a.x, b.x, c.x), fmaf(a.y, b.y, c.y), fmaf(a.z, b.z, c.z), fmaf(a.w, b.w, c.w)};
}
__device__ __forceinline__ V4 vaxpy(float c, V4 a, V4 b) {  // c a + b
    return V4{fmaf(c, a.x, b.x), fmaf(c, a.y, b.y), fmaf(c, a.z, b.z), fmaf(c, a.w, b.w)};
}
__device__ __forceinline__ float vmul(float a, float b) { return a * b; }
__device__ __forceinline__ float vscale(float c, float a) { return c * a; }
__device__ __forceinline__ float vfma(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ float vaxpy(float c, float a, float b) { return fmaf(c, a, b); }

template <class T>
__device__ __forceinline__ T v_central(T m2, T m1, T p1, T p2) {
    return vaxpy(-C_1_12, p2, vaxpy(C_2_3, p1, vaxpy(-C_2_3, m1, vscale(C_1_12, m2))));
}
template <class T>
__device__ __forceinline__ T v_head(T a, T b, T c, T d) {
    return vaxpy(C_1_3, d, vaxpy(-C_3_2, c, vaxpy(C_THREE, b, vscale(C_HEAD0, a))));
}
template <class T>
__device__ __forceinline__ T v_tail(T a, T b, T c, T d) {
    return vaxpy(C_TAIL3, d, vaxpy(-C_THREE, c, vaxpy(C_3_2, b, vscale(C_TAIL0, a))));
}

// One axis at R neighbouring cells x0 .. x0+R-1 of a line of N cells, in two halves so that few
// values are live at a time; derivatives unscaled (results times 1/dx^2).  EDGE: a cell of the warp
// lies within reach of one of the line's ends.  cell(f, d) is cell x0 + d of field f (0: u, 1: D, both
// edge-padded; 2: lambda_u, zero outside the grid); of(f, t) the same at d = t - 4 for the t known at
// compile time.  v_central with its arguments reversed is -G.
//
// gd: lambda u'' + B^T (lambda u').
template <int R, bool EDGE, class T, class Of, class At>
__device__ __forceinline__ void axis_gd(int x0, int N, Of of, At cell, T (&gd)[R]) {
    T U[R + 8], ux[R + 4];
#pragma unroll
    for (int t = 0; t < 4; ++t) U[t] = of(0, t);
#pragma unroll
    for (int t = 0; t < R + 4; ++t) {
        U[t + 4] = of(0, t + 4);
        ux[t] = v_central(U[t], U[t + 1], U[t + 3], U[t + 4]);
        if (EDGE) {
            const int x = x0 - 2 + t;
            if (t <= 2 && x <= 0) ux[t] = v_head(cell(0, t - 2), cell(0, t - 1), cell(0, t), cell(0, t + 1));
            if (t >= 1 && x >= N - 1) ux[t] = v_tail(cell(0, t - 5), cell(0, t - 4), cell(0, t - 3), cell(0, t - 2));
        }
    }
#pragma unroll
    for (int k = 0; k < R; ++k) {
        T d = v_central(ux[k], ux[k + 1], ux[k + 3], ux[k + 4]);
        if (EDGE) {
            const int x = x0 + k;
            if (k == 0 && x == 0) d = v_head(ux[2], ux[3], ux[4], ux[5]);
            if (x == N - 1) {
                T far = ux[k >= 1 ? k - 1 : 0];
                if (k == 0) far = v_central(cell(0, -5), cell(0, -4), cell(0, -2), cell(0, -1));
                d = v_tail(far, ux[k], ux[k + 1], ux[k + 2]);
            }
        }
        gd[k] = vmul(of(2, k + 4), d);
    }
    // lambda u', with the one-sided rows 0 and N-1 taken out of the central sums
    T (&m)[R + 4] = ux;
#pragma unroll
    for (int t = 0; t < R + 4; ++t) m[t] = vmul(of(2, t + 2), ux[t]);
    if (EDGE) {
        const T zero = vscale(0.0f, T{}), m1 = m[3];
        const int dn = N - 1 - x0;
        T m0 = zero, mn = zero;
        if (x0 <= 4) m0 = vmul(cell(2, -x0), v_head(cell(0, -x0), cell(0, 1 - x0), cell(0, 2 - x0), cell(0, 3 - x0)));
        if (dn <= R + 4) mn = vmul(cell(2, dn), v_tail(cell(0, dn - 3), cell(0, dn - 2), cell(0, dn - 1), cell(0, dn)));
#pragma unroll
        for (int t = 0; t < R + 4; ++t) {
            if (t < 3 && x0 - 2 + t <= 0) m[t] = zero;
            if (t >= 2 && x0 - 2 + t >= N - 1) m[t] = zero;
        }
#pragma unroll
        for (int k = 0; k < R; ++k) {
            const int x = x0 + k;
            gd[k] = vaxpy((unsigned)x < 4u ? kHeadC[x & 3] : 0.0f, m0, gd[k]);
            gd[k] = vaxpy(x >= N - 4 && x < N ? kTailC[(x - N) & 3] : 0.0f, mn, gd[k]);
            // the pad rows fold onto the first and the last cell
            if (k == 0 && x == 0) gd[k] = vaxpy(C_1_12, m1, gd[k]);
            if (x == N - 1) gd[k] = vaxpy(-C_1_12, m[k + 1], gd[k]);
        }
    }
#pragma unroll
    for (int k = 0; k < R; ++k) gd[k] = vaxpy(1.0f, v_central(m[k + 4], m[k + 3], m[k + 1], m[k]), gd[k]);
}

// at: A^T (D lambda) + B^T ((B D) lambda).
template <int R, bool EDGE, class T, class Of, class At>
__device__ __forceinline__ void axis_at(int x0, int N, Of of, At cell, T (&at)[R]) {
    const T zero = vscale(0.0f, T{});
    // D lambda at the one-sided rows (q0, qn), and what these rows and the pad rows carry into the
    // second operator (b0, bm and bn, bp)
    T q0 = zero, b0 = zero, bm = zero, qn = zero, bn = zero, bp = zero;
    if (EDGE) {
        if (x0 <= 4) {
            const int d = -x0;
            auto Q = [&](int k) { return vmul(cell(1, d + k), cell(2, d + k)); };
            q0 = Q(0);
            const T q1 = Q(1);
            bm = vscale(C_1_12, q1);
            const T g = v_head(cell(1, d), cell(1, d + 1), cell(1, d + 2), cell(1, d + 3));
            b0 = vfma(g, cell(2, d), vaxpy(C_HEAD0, q0, vaxpy(-C_2_3, q1, vscale(C_1_12, Q(2)))));
        }
        if (N - 1 - x0 <= R + 4) {
            const int d = N - 1 - x0;
            auto Q = [&](int k) { return vmul(cell(1, d - k), cell(2, d - k)); };
            qn = Q(0);
            const T q1 = Q(1);
            bp = vscale(-C_1_12, q1);
            const T g = v_tail(cell(1, d - 3), cell(1, d - 2), cell(1, d - 1), cell(1, d));
            bn = vfma(g, cell(2, d), vaxpy(C_TAIL3, qn, vaxpy(C_2_3, q1, vscale(-C_1_12, Q(2)))));
        }
    }
    T D[R + 8], q[R + 8], s[R + 4];
    auto take = [&](int t) {
        D[t] = of(1, t);
        q[t] = vmul(D[t], of(2, t));
        if (EDGE) {
            const int x = x0 - 4 + t;
            if ((t <= 4 && x == 0) || (t >= 4 && x == N - 1)) q[t] = zero;
        }
    };
#pragma unroll
    for (int t = 0; t < 4; ++t) take(t);
#pragma unroll
    for (int t = 0; t < R + 4; ++t) {
        take(t + 4);
        T g = v_central(D[t], D[t + 1], D[t + 3], D[t + 4]);
        T y = v_central(q[t + 4], q[t + 3], q[t + 1], q[t]);
        if (EDGE) {
            const int x = x0 - 2 + t;
            if (t <= 2 && x == 0) g = v_head(cell(1, t - 2), cell(1, t - 1), cell(1, t), cell(1, t + 1));
            if (t >= 1 && x == N - 1) g = v_tail(cell(1, t - 5), cell(1, t - 4), cell(1, t - 3), cell(1, t - 2));
            y = vaxpy((unsigned)x < 4u ? kHeadC[x & 3] : 0.0f, q0, y);
            y = vaxpy((unsigned)(x - N + 4) < 4u ? kTailC[(x - N) & 3] : 0.0f, qn, y);
        }
        s[t] = vfma(g, of(2, t + 2), y);
    }
    const T s1 = s[3];
    if (EDGE)  // rows -1, 0 and N-1, N leave the central sums of the second operator
#pragma unroll
        for (int t = 0; t < R + 4; ++t) {
            if (t < 3 && x0 - 2 + t <= 0) s[t] = zero;
            if (t >= 2 && x0 - 2 + t >= N - 1) s[t] = zero;
        }
#pragma unroll
    for (int k = 0; k < R; ++k) {
        T a = v_central(s[k + 4], s[k + 3], s[k + 1], s[k]);
        if (EDGE) {
            const int x = x0 + k;
            a = vaxpy((unsigned)x < 4u ? kHeadC[x & 3] : 0.0f, b0, a);
            a = vaxpy((unsigned)x < 3u ? kHeadC[(x + 1) & 3] : 0.0f, bm, a);
            a = vaxpy(x >= N - 4 && x < N ? kTailC[(x - N) & 3] : 0.0f, bn, a);
            a = vaxpy(x >= N - 3 && x < N ? kTailC[(x - N - 1) & 3] : 0.0f, bp, a);
            if (k == 0 && x == 0) a = vaxpy(C_HEAD0, bm, vaxpy(C_1_12, s1, a));  // the pad rows fold
            if (x == N - 1) a = vaxpy(C_TAIL3, bp, vaxpy(-C_1_12, s[k + 1], a));
        }
        at[k] = a;
    }
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

// Tile (bx, by) of an nbx x nby cut of the grid (rows in groups of LR, columns in quads, dealt out
// evenly; the last tile row's groups are aligned to the bottom, so that rows 0 and H-1 are the first
// and the last row of a thread).  Its dL/dtheta sums go to slot by * nbx + bx of a.gtheta.
__device__ __forceinline__ void adjoint_line_tile(const AdjointArgs &a, int bx, int by, int nbx,
                                                  int nby) {
    __shared__ __align__(16) float su[LSH * LSW];
    __shared__ __align__(16) float sd[LSH * LSW];
    __shared__ __align__(16) float sl[LSH * LSW];
    __shared__ float4 sp[4][LR][LU];  // a unit's own v, w, lambda_v, lambda_w; the first then its
                                      // lambda_u through the currents
    __shared__ float4 sr[2][LR][LU];  // the x direction's part of lambda_u and of dL/dD
    __shared__ float red[LU / 32][16];
    const int tid = threadIdx.x, lane = tid & 31;
    const int role = tid / LU, unit = tid % LU;
    const int H = a.H, W = a.W, pitch = a.pitch;
    const float dt = a.dt, rdx = a.rdx;
    const int ng = (H + LR - 1) / LR, nq = (W + 3) / 4;
    const int g0 = by * ng / nby, g1 = (by + 1) * ng / nby;
    const int c0 = bx * nq / nbx, c1 = (bx + 1) * nq / nbx;
    const int shift = by == nby - 1 ? ng * LR - H : 0;
    const int row0 = g0 * LR - shift, j0 = 4 * c0;   // the tile's first group's first row
    const int rows = (g1 - g0) * LR, tq = c1 - c0;
    // units by pairs of quad columns: those near the left and right sides then lie in few warps
    const int G = g1 - g0, pair = (unit >> 1) / G;
    const bool mine = 2 * pair + (unit & 1) < tq;
    const int lq = mine ? 2 * pair + (unit & 1) : 0, lg = mine ? (unit >> 1) - pair * G : 0;
    const int i0 = row0 + lg * LR, j = j0 + 4 * lq;
    const int k_lo = by == nby - 1 && lg == 0 ? shift : 0;  // rows before it belong to the tile above
    const int64_t off0 = (int64_t)i0 * pitch + j;

    // All reads go through L2: with programmatic dependent launch this block may have started before
    // the step that wrote lambda and dL/dD ended, and L1 is not coherent with the other SMs.
    // ---- stage u, D, lambda_u with 4 cells around: clamped copies outside the grid, lambda 0 ------
    constexpr int N4 = LSW / 4, RPP = LNT / N4;  // quads of a staged row, rows per pass
    if (tid < RPP * N4 && tid % N4 < tq + 2) {
        const int c = 4 * (tid % N4), jc = j0 - 4 + c;
        const bool quad_in = jc >= 0 && jc + 3 < W;
        for (int r = tid / N4; r < rows + 8; r += RPP) {
            const int i = row0 - 4 + r;
            const int64_t g = (int64_t)clampi(i, 0, H - 1) * pitch;
            const int o = r * LSW + c;
            const bool row_in = i >= 0 && i < H;
            if (quad_in) {
                cp_async16(su + o, a.u + g + jc);
                cp_async16(sd + o, a.D + g + jc);
                if (row_in) cp_async16(sl + o, a.lu + g + jc);
                else *reinterpret_cast<float4 *>(sl + o) = make_float4(0.f, 0.f, 0.f, 0.f);
            } else {
                // a quad across or beyond the grid's side: the nearest cell in place of those outside
                const int jn = clampi(jc, 0, 4 * (nq - 1));  // the quad of the row that has it
                float4 x = __ldcg(reinterpret_cast<const float4 *>(a.u + g + jn));
                float4 y = __ldcg(reinterpret_cast<const float4 *>(a.D + g + jn));
                float4 z = __ldcg(reinterpret_cast<const float4 *>(a.lu + g + jn));
                if (jc < 0) {
                    x.y = x.z = x.w = x.x;
                    y.y = y.z = y.w = y.x;
                }
                const int n = W - 1 - jn;  // the last cell's place in the quad
                if (n < 1) x.y = x.x, y.y = y.x;
                if (n < 2) x.z = x.y, y.z = y.y;
                if (n < 3) x.w = x.z, y.w = y.z;
                if (jc > jn) {
                    x.x = x.y = x.z = x.w;
                    y.x = y.y = y.z = y.w;
                }
                const bool l_in = row_in && jc == jn;
                z.x = l_in ? z.x : 0.0f;
                z.y = l_in && n >= 1 ? z.y : 0.0f;
                z.z = l_in && n >= 2 ? z.z : 0.0f;
                z.w = l_in && n >= 3 ? z.w : 0.0f;
                *reinterpret_cast<float4 *>(su + o) = x;
                *reinterpret_cast<float4 *>(sd + o) = y;
                *reinterpret_cast<float4 *>(sl + o) = z;
            }
        }
    }
    if (role == 0)
#pragma unroll
        for (int k = 0; k < LR; ++k)
            if (mine && k >= k_lo) {
                const int64_t o = off0 + (int64_t)k * pitch;  // j < W: the quad lies in the pitched row
                cp_async16(reinterpret_cast<float *>(&sp[0][k][unit]), a.v + o);
                cp_async16(reinterpret_cast<float *>(&sp[1][k][unit]), a.w + o);
                cp_async16(reinterpret_cast<float *>(&sp[2][k][unit]), a.lv + o);
                cp_async16(reinterpret_cast<float *>(&sp[3][k][unit]), a.lw + o);
            } else {
#pragma unroll
                for (int f = 0; f < 4; ++f) sp[f][k][unit] = make_float4(0.f, 0.f, 0.f, 0.f);
            }
    const unsigned active = __ballot_sync(0xffffffffu, lane < a.n_stim && stim_active(a.stim[lane < kMaxStim ? lane : 0], a.t));
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();

    double *const slot = a.gtheta + (int64_t)(by * nbx + bx) * kAdjParamStride + (tid < 12 ? tid : 0);
    const double slot_was = a.gtheta && tid < 12 ? __ldcg(slot) : 0.0;  // early: its trip overlaps the work

    // Role 0 takes the pointwise part, role 1 the x direction (along rows), of the unit's two rows;
    // then the y direction of row 0 and of row 1: the chain of one thread is half as long.
    const int base = (lg * LR + 4) * LSW + 4 * lq + 4;  // the unit's first cell
    if (role == 0) {
        const Model &md = a.m;
        float gth[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) gth[k] = 0.0f;
#pragma unroll 1
        for (int k = 0; k < LR; ++k) {
            const float4 v4 = sp[0][k][unit], w4 = sp[1][k][unit];
            float4 lv4 = sp[2][k][unit], lw4 = sp[3][k][unit];
            const float4 u4 = *reinterpret_cast<const float4 *>(su + base + k * LSW);
            const float4 l4 = *reinterpret_cast<const float4 *>(sl + base + k * LSW);
            float4 lj4 = l4;  // lambda_u where the current is the model's
            const int i = i0 + k;
            const int64_t o = off0 + (int64_t)k * pitch;
            const bool row_ok = mine && k >= k_lo;
            if (!row_ok) lj4 = make_float4(0.f, 0.f, 0.f, 0.f);
            if (j + 3 >= W) {  // columns beyond W (lambda_u is zero there)
                if (j + 1 >= W) lv4.y = lw4.y = 0.f;
                if (j + 2 >= W) lv4.z = lw4.z = 0.f;
                lv4.w = j + 3 >= W ? 0.f : lv4.w;
                lw4.w = j + 3 >= W ? 0.f : lw4.w;
            }
            if (active && row_ok)  // cells whose current a stimulus replaces
                for (unsigned x = active; x; x &= x - 1) {
                    const Stim &st = a.stim[__ffs(x) - 1];
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
                    if (f.x != 0.0f) lj4.x = 0.0f;
                    if (f.y != 0.0f) lj4.y = 0.0f;
                    if (f.z != 0.0f) lj4.z = 0.0f;
                    if (f.w != 0.0f) lj4.w = 0.0f;
                }
            const float uu[4] = {u4.x, u4.y, u4.z, u4.w}, ll[4] = {l4.x, l4.y, l4.z, l4.w};
            const float vv[4] = {v4.x, v4.y, v4.z, v4.w}, ww[4] = {w4.x, w4.y, w4.z, w4.w};
            const float lvv[4] = {lv4.x, lv4.y, lv4.z, lv4.w}, lww[4] = {lw4.x, lw4.y, lw4.z, lw4.w};
            const float ljj[4] = {lj4.x, lj4.y, lj4.z, lj4.w};
            float ov[4], ow[4], pu[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const float u = uu[c], v = vv[c], w = ww[c], lv = lvv[c], lw = lww[c], lj = ljj[c];
                const bool p = u >= md.V_c, q = u >= md.V_v;
                const float uk = u - md.V_csi;
                const float S = one_plus_tanh(md.k * uk);  // 1 + tanh
                const float sech2 = S * (2.0f - S);        // 1 - tanh^2
                const float uc = u - md.V_c, u1 = 1.0f - u;
                // (as one product with 1 + dt x, its rounding would act the same way in every step: dL/dv0
                // off by up to 6e-8 per step)
                ov[c] = fmaf(lv, dt * (p ? -md.r_tau_vp : (q ? -md.r_tau_v2m : -md.r_tau_v1m)), lv);
                ow[c] = fmaf(lw, dt * (p ? -md.r_tau_wp : -md.r_tau_wm), lw);
                const float dfi = p ? -v * (1.0f + md.V_c - 2.0f * u) * md.r_tau_d : 0.0f;
                const float dso = p ? 0.0f : md.r_tau_0;
                const float dsi = -w * md.k * sech2 * md.r_2tau_si;
                const float mu = dt * lj;
                ov[c] = fmaf(mu, p ? uc * u1 * md.r_tau_d * md.r_Cm : 0.0f, ov[c]);
                ow[c] = fmaf(mu, S * md.r_2tau_si * md.r_Cm, ow[c]);
                pu[c] = fmaf(mu, -(dfi + dso + dsi) * md.r_Cm, ll[c]);
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
            if (row_ok) {
                if (j + 3 < W) {
                    *reinterpret_cast<float4 *>(a.olv + o) = make_float4(ov[0], ov[1], ov[2], ov[3]);
                    *reinterpret_cast<float4 *>(a.olw + o) = make_float4(ow[0], ow[1], ow[2], ow[3]);
                } else {
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        if (j + c < W) {
                            a.olv[o + c] = ov[c];
                            a.olw[o + c] = ow[c];
                        }
                }
            }
        }
        if (a.gtheta) {
            const float x = warp_sum16(gth);
            if (lane < 16) red[unit / 32][lane] = x;
        }
    } else {
        V4 x[LR];
        auto cell = [&](int f, int d) {
            return ld_v4((f == 0 ? su : f == 1 ? sd : sl) + base + d * LSW);
        };
        auto of = [&](int f, int t) { return cell(f, t - 4); };
        const bool edge = __any_sync(0xffffffffu, mine && (i0 <= 5 || i0 + LR + 1 >= H - 4)) != 0;
        if (edge) axis_gd<LR, true, V4>(i0, H, of, cell, x);
        else axis_gd<LR, false, V4>(i0, H, of, cell, x);
#pragma unroll
        for (int k = 0; k < LR; ++k) sr[1][k][unit] = make_float4(x[k].x, x[k].y, x[k].z, x[k].w);
        if (edge) axis_at<LR, true, V4>(i0, H, of, cell, x);
        else axis_at<LR, false, V4>(i0, H, of, cell, x);
#pragma unroll
        for (int k = 0; k < LR; ++k) sr[0][k][unit] = make_float4(x[k].x, x[k].y, x[k].z, x[k].w);
    }
    const int k = role;  // LR == 2
    const bool stored = mine && k >= k_lo;
    const int64_t g = off0 + (int64_t)k * pitch;
    float4 gd4 = make_float4(0.f, 0.f, 0.f, 0.f);
    if (a.gD && stored) gd4 = __ldcg(reinterpret_cast<const float4 *>(a.gD + g));
    float ay[4], gy[4];
    {
        const int o = base + k * LSW;
        auto cell = [&](int f, int d) { return (f == 0 ? su : f == 1 ? sd : sl)[o + d]; };
        float L[12], F[12];
        auto row = [&](const float *p, float (&x)[12]) {
#pragma unroll
            for (int t = 0; t < 3; ++t) {
                const float4 y = *reinterpret_cast<const float4 *>(p + o + 4 * t - 4);
                x[4 * t] = y.x, x[4 * t + 1] = y.y, x[4 * t + 2] = y.z, x[4 * t + 3] = y.w;
            }
        };
        row(sl, L);
        row(su, F);
        auto of = [&](int f, int t) { return f == 2 ? L[t] : F[t]; };
        const bool edge = __any_sync(0xffffffffu, mine && (j <= 5 || j + 5 >= W - 4)) != 0;
        if (edge) axis_gd<4, true, float>(j, W, of, cell, gy);
        else axis_gd<4, false, float>(j, W, of, cell, gy);
        row(sd, F);
        if (edge) axis_at<4, true, float>(j, W, of, cell, ay);
        else axis_at<4, false, float>(j, W, of, cell, ay);
    }
    __syncthreads();
    if (stored) {
        const float c2 = rdx * rdx * dt;
        const float4 pu = sp[0][k][unit], ax = sr[0][k][unit], gx = sr[1][k][unit];
        const float4 r = make_float4(fmaf(c2, ax.x + ay[0], pu.x), fmaf(c2, ax.y + ay[1], pu.y),
                                     fmaf(c2, ax.z + ay[2], pu.z), fmaf(c2, ax.w + ay[3], pu.w));
        gd4 = make_float4(fmaf(c2, gx.x + gy[0], gd4.x), fmaf(c2, gx.y + gy[1], gd4.y),
                          fmaf(c2, gx.z + gy[2], gd4.z), fmaf(c2, gx.w + gy[3], gd4.w));
        if (j + 3 < W) {
            *reinterpret_cast<float4 *>(a.olu + g) = r;
            if (a.gD) __stcg(reinterpret_cast<float4 *>(a.gD + g), gd4);
        } else {
            const float rr[4] = {r.x, r.y, r.z, r.w}, ee[4] = {gd4.x, gd4.y, gd4.z, gd4.w};
#pragma unroll
            for (int c = 0; c < 4; ++c)
                if (j + c < W) {
                    a.olu[g + c] = rr[c];
                    if (a.gD) __stcg(a.gD + g + c, ee[c]);
                }
        }
    }
    if (a.gtheta && tid < 12) {
        double x = 0.0;
#pragma unroll
        for (int w = 0; w < LU / 32; ++w) x += (double)red[w][tid];
        __stcg(slot, fma(a.theta_factor[tid], x, slot_was));
    }
}

__global__ void __launch_bounds__(LNT, 2) fk_adjoint_line_kernel(const __grid_constant__ AdjointArgs a) {
    grid_dependency_wait();
    grid_launch_dependents();
    adjoint_line_tile(a, blockIdx.x, blockIdx.y, gridDim.x, gridDim.y);
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

__global__ void __launch_bounds__(LNT, 2)
    fk_adjoint_line_batch_kernel(const AdjointArgs *__restrict__ exps, int64_t k_stride, int k,
                                 int parity, float t) {
    __shared__ __align__(16) AdjointArgs sa;
    grid_dependency_wait();
    grid_launch_dependents();
    stage_experiment(sa, exps, k_stride, k, parity, t);
    adjoint_line_tile(sa, blockIdx.x, blockIdx.y, gridDim.x, gridDim.y);
}

// Which kernel takes a grid, and its blocks.
bool long_lines(int H, int W) { return H >= kLineMin && W >= kLineMin; }
dim3 adjoint_grid(int H, int W, int n_exp) {
    if (!long_lines(H, W)) return dim3((W + ATX - 1) / ATX, (H + ATY - 1) / ATY, n_exp);
    return dim3(((W + 3) / 4 + LQ - 1) / LQ, ((H + LR - 1) / LR + LG - 1) / LG, n_exp);
}

template <class K, class... A>
cudaError_t launch_line(K kernel, dim3 grid, cudaStream_t stream, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(LNT);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
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
    const dim3 g = adjoint_grid(H, W, 1);
    return (int64_t)g.x * g.y;
}

cudaError_t launch_adjoint(const AdjointArgs &a, cudaStream_t stream) {
    const dim3 grid = adjoint_grid(a.H, a.W, 1);
    if (long_lines(a.H, a.W)) return launch_line(fk_adjoint_line_kernel, grid, stream, a);
    fk_adjoint_kernel<<<grid, ANT, 0, stream>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_adjoint_batch(const AdjointArgs *exps, int n_exp, int H, int W, int64_t k_stride,
                                 int k, int parity, float t, cudaStream_t stream) {
    if (n_exp < 1) return cudaSuccess;
    const dim3 grid = adjoint_grid(H, W, n_exp);
    if (long_lines(H, W))
        return launch_line(fk_adjoint_line_batch_kernel, grid, stream, exps, k_stride, k, parity, t);
    fk_adjoint_batch_kernel<<<grid, ANT, 0, stream>>>(exps, k_stride, k, parity, t);
    return cudaGetLastError();
}

}  // namespace fk
