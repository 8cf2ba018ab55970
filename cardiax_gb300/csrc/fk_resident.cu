// K8: the resident stepper -- many Euler steps of a small or mid-sized tissue in one cooperative
// launch with the whole state on chip (cardiax/solve.py:92-100, _forward_euler).
//
// One CTA per SM owns one tile of the grid for the whole launch.  A thread owns R rows of one quad
// of columns: v and w stay in its registers, D and its two slopes (constant over the launch) in
// shared memory, and u in a double-buffered shared-memory tile with a 4-cell halo.  Per step a
// thread reads the u rows around its cells, forms u_x and u_y in registers (no second pass) and
// updates its cells; then the cells within 4 of a tile side go to the neighbour through global
// memory.  Only u is exchanged, only with the 4 direct neighbours: no stencil is diagonal.
//
// What bounds it (us per step, GB300; one launch per step before): 256^2 1.84 (4.4), 512^2 2.36
// (4.5), 1024^2 5.08 (8.2), 1200^2 5.97 (9.7).  One launch per step pays launch, load and store
// latencies in a row whatever it computes.  Here a small grid's step is one dependent chain: about
// 1000 cycles for a unit of 8 cells (1600 at the grid's edge), 1700 from a strip's store to its
// neighbour's load of it through L2, and two barriers.  A large grid's step is bound by issue
// slots and instruction fetch (some 89 instructions per cell); the loop's code is kept small for that
// reason (see Unit).
//
// Rows per thread: more rows share u rows and u_x, and hold more cells (512 threads of 4 R cells
// on each SM: 152 SMs hold 1247^2 cells at R = 5), but lengthen the chain: a 256^2 step takes
// 1.8 / 2.5 / 3.4 / 4.3 us at R = 2 / 3 / 4 / 5, so resident_plan takes the fewest that fit.
//
// The exchange.  A word of a strip is 8 bytes, (float, step tag), stored and loaded as one 64-bit
// access, so a reader that sees the tag of the step it waits for has the value as well: no flag,
// no fence, one store-to-load trip through L2 per step.  Two buffers (step parity) suffice: a tile
// overwrites the strip of step s at step s + 2, after it has read its neighbours' strips of step
// s + 1, which they sent after they had read its strip of step s.
//
// A tissue of few cells per SM on 16 SMs runs as one cluster instead: the strips are stored straight into the
// neighbours' u tiles (distributed shared memory) and the cluster's barrier takes the place of the tags; no
// words in memory, no spinning, no cooperative launch.  64^2 1.88 -> 1.57 us per step, 128^2 1.88 -> 1.62.
//
// Every wait on memory is bounded (1 s); a tile whose wait runs out reports it and leaves, its neighbours'
// waits then run out as well.  The launch is cooperative, so all tiles run at the same time, and
// takes at most kResMaxSteps steps.
//
// Several tissues (MANY): each CTA finds its tissue in a table and takes that tissue's plan, constants
// and buffers; the tissues of a launch share rows per thread and CTA size and nothing else.
//
// Per cell these are the operations of the step kernel in the same order (fk_pack.cuh): the same
// bits.
#include "fk_resident.cuh"

#include "fk_capi_internal.h"
#include "fk_tile.cuh"

namespace fk {

namespace {

__device__ __forceinline__ void st_tagged(uint64_t *p, float a, float b, uint32_t tag) {
    const uint64_t t = (uint64_t)tag << 32;
    const uint64_t x = t | __float_as_uint(a), y = t | __float_as_uint(b);
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(x), "l"(y) : "memory");
}
__device__ __forceinline__ void ld_tagged(const uint64_t *p, uint64_t &x, uint64_t &y) {
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(x), "=l"(y) : "l"(p) : "memory");
}
// The other CTAs of the cluster: an address of theirs for one of this CTA's, a store there, and the barrier
// (arrive releases this CTA's stores, wait acquires the others').
__device__ __forceinline__ uint32_t cluster_addr(const float *p, int rank) {
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_addr(p)), "r"(rank));
    return a;
}
__device__ __forceinline__ void st_cluster(uint32_t a, float4 q) {
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(q.x), "f"(q.y), "f"(q.z), "f"(q.w)
                 : "memory");
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
// A quad of a strip: two 16-byte accesses.
__device__ __forceinline__ void send_quad(uint64_t *p, float4 q, uint32_t tag) {
    st_tagged(p, q.x, q.y, tag);
    st_tagged(p + 2, q.z, q.w, tag);
}
__device__ __forceinline__ bool try_quad(const uint64_t *p, uint32_t tag, float4 &q) {
    uint64_t a, b, c, d;
    ld_tagged(p, a, b);
    ld_tagged(p + 2, c, d);
    q = make_float4(__uint_as_float((uint32_t)a), __uint_as_float((uint32_t)b),
                    __uint_as_float((uint32_t)c), __uint_as_float((uint32_t)d));
    return (uint32_t)(a >> 32) == tag && (uint32_t)(b >> 32) == tag &&
           (uint32_t)(c >> 32) == tag && (uint32_t)(d >> 32) == tag;
}
// Waits for a quad of step `tag`, at most 1 s.  (Several loads kept in flight, staggered, to see
// the quad sooner after it arrives measured no faster: 2.27 against 2.35 us per 256^2 step, 6.9
// against 6.5 at 1200^2.)
__device__ __forceinline__ bool wait_quad(const uint64_t *p, uint32_t tag, float4 &q) {
    if (try_quad(p, tag, q)) return true;
    const uint64_t t0 = global_timer_ns();
    for (;;) {
        for (int k = 0; k < 64; ++k)
            if (try_quad(p, tag, q)) return true;
        if (global_timer_ns() - t0 > 1000000000ull) return false;
    }
}

// The first slope (scaled) at cell x of a line of N cells, p its place in an edge-padded tile with
// `stride` floats from one cell of the line to the next.
__device__ __forceinline__ float slope(const float *p, int stride, int x, int N, float rdx) {
    float s;
    if (x == 0) s = g_head(p[0], p[stride], p[2 * stride], p[3 * stride]);
    else if (x == N - 1) s = g_tail(p[-3 * stride], p[-2 * stride], p[-stride], p[0]);
    else s = g_central(p[-2 * stride], p[-stride], p[stride], p[2 * stride]);
    return s * rdx;
}

// Stimulus override of the 4 ionic currents of cells (i, j .. j+3): later active stimuli win, a
// zero value leaves the current (cardiax/solve.py:257-271).
__device__ __forceinline__ void override_current(const StepArgs &a, unsigned active, int i, int j,
                                                 int64_t goff, float2 &lo, float2 &hi) {
    for (unsigned on = active; on; on &= on - 1) {
        const Stim &st = a.stim[__ffs(on) - 1];
        float4 f;
        if (st.field) {
            f = __ldg(reinterpret_cast<const float4 *>(st.field + goff));
        } else {
            const bool in = i >= st.r0 && i < st.r1;
            f.x = in && j >= st.c0 && j < st.c1 ? st.amplitude : 0.0f;
            f.y = in && j + 1 >= st.c0 && j + 1 < st.c1 ? st.amplitude : 0.0f;
            f.z = in && j + 2 >= st.c0 && j + 2 < st.c1 ? st.amplitude : 0.0f;
            f.w = in && j + 3 >= st.c0 && j + 3 < st.c1 ? st.amplitude : 0.0f;
        }
        if (f.x != 0.0f) lo.x = f.x;
        if (f.y != 0.0f) lo.y = f.y;
        if (f.z != 0.0f) hi.x = f.z;
        if (f.w != 0.0f) hi.y = f.w;
    }
}

// on ? a : b with both computed (written as a conditional the compiler moves the computation of
// `a` into a branch, and a divergent branch costs more than the four instructions it skips).
__device__ __forceinline__ float pick(int on, float a, float b) {
    float d;
    asm("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %3, 0;\n\tselp.f32 %0, %1, %2, p;\n\t}"
        : "=f"(d)
        : "f"(a), "f"(b), "r"(on));
    return d;
}

// A thread's unit and where it lies.
struct Unit {
    int i0, j;         // its first row and column
    int k_lo;          // its first row that belongs to this tile (nonzero in the last tile row only)
    int64_t off0;      // i0 * pitch + j
    // whether a unit of this warp meets column 0, column W-1, row 0, row H-1 (warp-uniform: warps
    // that do not skip the one-sided rows and columns; one code path for all keeps the loop's
    // instructions in the instruction cache, two paths measured twice as slow where both ran)
    bool left, right, top, bottom;
};

// The tissue's constants: of the launch's one tissue, or of this block's class.
struct Consts {
    const Model &m;
    float rdx, dt;
    float2 rdx2, dt2;  // each twice
};

// One step of a unit: reads u around it at `c` (its first cell in the current buffer), writes the
// new u to `dst` (the same place in the next one) and updates v and w in place.
template <int R, bool ACT>
__device__ __forceinline__ void step_unit(const StepArgs &a, const Consts &tc, const PackConsts &kc,
                                          const Unit &un, const float *c, float *dst, int SUW,
                                          const float4 *sD, int nthr, float4 (&v)[R],
                                          float4 (&w)[R], unsigned active, float t) {
    const int H = a.H, W = a.W;
    const float rdx = tc.rdx;
    const int i0 = un.i0, j = un.j;
    // u rows -4+q and u_x rows -2+q of this quad, relative to its first row, taken as needed
    Quad U[R + 8], X[R + 4];
    auto take_u = [&](int q) { U[q] = ld_quad(c + (q - 4) * SUW); };
    auto take_x = [&](int q) {
        X[q] = q_central(kc, U[q], U[q + 1], U[q + 3], U[q + 4]);
        // The one-sided rows -1, 0 and H-1, H.  Rows 0 and H-1 are the first and the last row of
        // a unit, so they fall on q = 1, 2 and R + 1, R + 2 (and, when units have two rows, on
        // q = 0 and R + 3 of the units beside those).
        if ((q == 1 || q == 2 || (R == 2 && q == 0)) && un.top)
            if (i0 - 2 + q <= 0) X[q] = q_head(kc, U[q + 2], U[q + 3], U[q + 4], U[q + 5]);
        if ((q == R + 1 || q == R + 2 || (R == 2 && q == R + 3)) && un.bottom)
            if (i0 - 2 + q >= H - 1) X[q] = q_tail(kc, U[q >= 1 ? q - 1 : 0], U[q], U[q + 1], U[q + 2]);
        X[q] = q_scale(X[q], tc.rdx2);
    };
#pragma unroll
    for (int q = 0; q < 8; ++q) take_u(q);
#pragma unroll
    for (int q = 0; q < 4; ++q) take_x(q);
#pragma unroll
    for (int k = 0; k < R; ++k) {
        const int i = i0 + k;
        take_u(k + 8);
        take_x(k + 4);
        Quad uxx = q_central(kc, X[k], X[k + 1], X[k + 3], X[k + 4]);
        if (k == 0 && un.top)
            if (i == 0) {  // u_x row 3 is not taken yet
                const Quad x3 = q_scale(q_central(kc, U[5], U[6], U[8], ld_quad(c + 5 * SUW)), tc.rdx2);
                uxx = q_head(kc, X[2], X[3], X[4], x3);
            }
        if (k == R - 1 && un.bottom)
            if (i == H - 1) uxx = q_tail(kc, X[k >= 1 ? k - 1 : 0], X[k], X[k + 1], X[k + 2]);
        uxx = q_scale(uxx, tc.rdx2);
        const Quad uc = U[k + 4];
        const float4 el = ld4(c + k * SUW - 4), er = ld4(c + k * SUW + 4);
        const float e[12] = {el.x,    el.y,    el.z, el.w, uc.lo.x, uc.lo.y,
                             uc.hi.x, uc.hi.y, er.x, er.y, er.z,    er.w};
        // u_y at columns j-2 .. j+5 as the pairs y[0] .. y[3]
        float2 y[4];
#pragma unroll
        for (int m = 0; m < 4; ++m)
            y[m] = pg_central_row(kc, e[2 * m], e[2 * m + 1], e[2 * m + 2], e[2 * m + 3], e[2 * m + 4],
                                  e[2 * m + 5]);
        // the one-sided columns -1, 0 (m = 1, 2 of j - 2 + m when j = 0) and W-1, W
        if (un.left) {
            y[0].y = pick(j == 0, g_head(e[3], e[4], e[5], e[6]), y[0].y);
            y[1].x = pick(j == 0, g_head(e[4], e[5], e[6], e[7]), y[1].x);
        }
        const int n = W - 1 - j;
        if (un.right) {
            const unsigned at = n <= 5 ? 3u << (n + 2) : 0u;  // bit m: column W-1 or W
#pragma unroll
            for (int m = 2; m < 8; ++m) {
                const float g = g_tail(e[m - 1], e[m], e[m + 1], e[m + 2]);
                if (m & 1) y[m / 2].y = pick(at & (1u << m), g, y[m / 2].y);
                else y[m / 2].x = pick(at & (1u << m), g, y[m / 2].x);
            }
        }
#pragma unroll
        for (int m = 0; m < 4; ++m) y[m] = p_mul(y[m], tc.rdx2);
        float2 yy_lo = pg_central_row(kc, y[0].x, y[0].y, y[1].x, y[1].y, y[2].x, y[2].y);
        float2 yy_hi = pg_central_row(kc, y[1].x, y[1].y, y[2].x, y[2].y, y[3].x, y[3].y);
        if (un.left) yy_lo.x = pick(j == 0, g_head(y[1].x, y[1].y, y[2].x, y[2].y), yy_lo.x);
        if (un.right) {
            // the tail's four u_y end at column W-1; at n = 0 the first one, at column j-3, lies
            // outside the window (a tile has two quads, so column j-5 is in shared memory when n = 0)
            const float ym = g_central(c[k * SUW - 5], e[0], e[2], e[3]) * rdx;
            yy_lo.x = pick(n == 0, g_tail(ym, y[0].x, y[0].y, y[1].x), yy_lo.x);
            yy_lo.y = pick(n == 1, g_tail(y[0].x, y[0].y, y[1].x, y[1].y), yy_lo.y);
            yy_hi.x = pick(n == 2, g_tail(y[0].y, y[1].x, y[1].y, y[2].x), yy_hi.x);
            yy_hi.y = pick(n == 3, g_tail(y[1].x, y[1].y, y[2].x, y[2].y), yy_hi.y);
        }
        yy_lo = p_mul(yy_lo, tc.rdx2);
        yy_hi = p_mul(yy_hi, tc.rdx2);
        const Quad d = ld_quad(reinterpret_cast<const float *>(sD + (0 * R + k) * nthr));
        const Quad dx = ld_quad(reinterpret_cast<const float *>(sD + (1 * R + k) * nthr));
        const Quad dy = ld_quad(reinterpret_cast<const float *>(sD + (2 * R + k) * nthr));
        const Reaction r0 = reaction(uc.lo.x, v[k].x, w[k].x, tc.m);
        const Reaction r1 = reaction(uc.lo.y, v[k].y, w[k].y, tc.m);
        const Reaction r2 = reaction(uc.hi.x, v[k].z, w[k].z, tc.m);
        const Reaction r3 = reaction(uc.hi.y, v[k].w, w[k].w, tc.m);
        float2 j_lo = mk2(r0.j_ion, r1.j_ion), j_hi = mk2(r2.j_ion, r3.j_ion);
        const int64_t goff = un.off0 + (int64_t)k * a.pitch;
        if (active && k >= un.k_lo) override_current(a, active, i, j, goff, j_lo, j_hi);
        // as in the step kernel: no packed multiply feeds a packed add
        float2 du_lo = p_mul(d.lo, add_products(uxx.lo, yy_lo));
        du_lo = p_fma(dx.lo, X[k + 2].lo, du_lo);
        du_lo = p_fma(dy.lo, y[1], du_lo);
        du_lo = p_add_product(kc, du_lo, j_lo);
        float2 du_hi = p_mul(d.hi, add_products(uxx.hi, yy_hi));
        du_hi = p_fma(dx.hi, X[k + 2].hi, du_hi);
        du_hi = p_fma(dy.hi, y[2], du_hi);
        du_hi = p_add_product(kc, du_hi, j_hi);
        const float dt = tc.dt;
        v[k] = make_float4(fmaf(r0.dv, dt, v[k].x), fmaf(r1.dv, dt, v[k].y), fmaf(r2.dv, dt, v[k].z),
                           fmaf(r3.dv, dt, v[k].w));
        w[k] = make_float4(fmaf(r0.dw, dt, w[k].x), fmaf(r1.dw, dt, w[k].y), fmaf(r2.dw, dt, w[k].z),
                           fmaf(r3.dw, dt, w[k].w));
        const float2 u_lo = p_fma(du_lo, tc.dt2, uc.lo), u_hi = p_fma(du_hi, tc.dt2, uc.hi);
        const bool stored = k >= un.k_lo;
        float4 u4 = make_float4(u_lo.x, u_lo.y, u_hi.x, u_hi.y);
        if (ACT) {
            const float uo4[4] = {uc.lo.x, uc.lo.y, uc.hi.x, uc.hi.y};
            const float un4[4] = {u4.x, u4.y, u4.z, u4.w};
#pragma unroll
            for (int m = 0; m < 4; ++m)
                if (stored && j + m < W) record_activation(a, t, goff + m, uo4[m], un4[m]);
        }
        float *o = dst + k * SUW;
        if (un.right) {  // the columns beyond W hold the edge padding
            u4.y = pick(n < 1, u4.x, u4.y);
            u4.z = pick(n < 2, u4.y, u4.z);
            u4.w = pick(n < 3, u4.z, u4.w);
            if (n == 3 && stored) o[4] = u4.w;
        }
        // one cell of padding beyond the grid on the other sides
        if (un.left)
            if (j == 0 && stored) o[-1] = u4.x;
        if (k == 0 && un.top)
            if (i == 0) st4(o - SUW, u4);
        if (k == R - 1 && un.bottom)
            if (i == H - 1) st4(o + SUW, u4);
        if (stored) st4(o, u4);
    }
}

}  // namespace

// R: rows per thread.  ACT: activation tracking.  MANY: the launch holds several tissues; ra.cta says
// which tissue (of ra.tissues) and which class of constants (ra.cls) a block belongs to.  Both are read
// from the launch's parameters by the block index, so the model's constants stay uniform operands.
// CL: the tiles are one thread-block cluster, their rank in it their number.
template <int R, bool ACT, bool MANY, bool CL>
__global__ void __launch_bounds__(512, 1)
    fk_resident_kernel(const __grid_constant__ ResidentArgs ra, const __grid_constant__ StepArgs a0,
                       const __grid_constant__ PackConsts kc) {
    extern __shared__ __align__(16) unsigned char res_smem[];
    __shared__ unsigned s_active[64];
    __shared__ int s_abort;  // a neighbour's strip did not come in time
    __shared__ __align__(16) unsigned char s_tissue[MANY ? sizeof(ResTissue) : 16];

    const int tid = threadIdx.x, nthr = blockDim.x;
    const uint32_t cta = MANY ? ra.cta[blockIdx.x] : 0u;
    if (MANY) {
        const uint32_t *src = reinterpret_cast<const uint32_t *>(ra.tissues + (cta >> 8));
        for (int k = tid; k < (int)(sizeof(ResTissue) / 4); k += nthr)
            reinterpret_cast<uint32_t *>(s_tissue)[k] = __ldg(src + k);
        __syncthreads();
    }
    const ResTissue &tis = *reinterpret_cast<const ResTissue *>(s_tissue);
    const StepArgs &a = MANY ? tis.args : a0;
    const ResClass &cls = ra.cls[MANY ? cta & 255u : 0];
    const Consts tconst{MANY ? cls.m : a0.m, MANY ? cls.rdx : a0.rdx, MANY ? cls.dt : a0.dt,
                        MANY ? mk2(cls.rdx, cls.rdx) : kc.rdx, MANY ? mk2(cls.dt, cls.dt) : kc.dt};
    const int H = a.H, W = a.W, pitch = a.pitch;
    const float rdx = tconst.rdx;
    const int t_nr = MANY ? tis.nr : ra.nr, t_nc = MANY ? tis.nc : ra.nc;
    const int t_ng = MANY ? tis.ng : ra.ng, t_nq = MANY ? tis.nq : ra.nq;
    const int tile = (int)blockIdx.x - (MANY ? tis.first : 0);
    const int tr = tile / t_nc, tc = tile % t_nc;
    const int g0 = tr * t_ng / t_nr, g1 = (tr + 1) * t_ng / t_nr;
    const int q0 = tc * t_nq / t_nc, q1 = (tc + 1) * t_nq / t_nc;
    const int row0 = g0 * R, row1 = tr == t_nr - 1 ? H : g1 * R;
    const int th = row1 - row0, tq = q1 - q0, j0 = 4 * q0;
    // The last tile row's groups are aligned to its bottom (so that row H-1 is the last row of a
    // thread and row 0 the first): its first group may reach `shift` rows above the tile, rows
    // that belong to the tile above and are not stored here.
    const int shift = g1 * R - row1 < 0 ? 0 : g1 * R - row1;
    const int SUW = MANY ? tis.su_w : ra.su_w, SU = ra.su;
    const int units = (g1 - g0) * tq;
    float *su = reinterpret_cast<float *>(res_smem);  // [2][su_h][su_w]: row r, column c at
    constexpr int UROW = 4 + R - 1, UCOL = 4;          // (r + UROW) * SUW + c + UCOL
    float4 *sD = reinterpret_cast<float4 *>(su + 2 * SU);  // [3][R][nthr]: D, D_x, D_y

    // This thread's unit: quad lq of row group lg.  The units at the tile's sides come first, the
    // left and right columns together, then the top and bottom rows: the units that meet the
    // grid's edge or the neighbours' cells then fill as few warps as they can.
    const bool mine = tid < units;
    const int G = g1 - g0;
    // groups that read the halo rows above and below the tile
    const int gt = min(G, (4 + shift + R - 1) / R), gb = min(G - gt, (4 + R - 1) / R);
    int lg = 0, lq = 0;
    if (tid < 2 * G) {
        lg = tid < G ? tid : tid - G;
        lq = tid < G ? 0 : tq - 1;
    } else if (mine) {  // tq > 2
        const int x = tid - 2 * G, y = x / (tq - 2);
        lq = 1 + x - y * (tq - 2);
        lg = y < gt ? y : (y < gt + gb ? G - 1 - (y - gt) : y - gb);
    }
    const int lr = lg * R - shift, lc = 4 * lq;
    const int i0 = row0 + lr, j = j0 + lc;
    const int64_t off0 = (int64_t)i0 * pitch + j;
    const int k_lo = lr < 0 ? -lr : 0;  // first row of the unit that belongs to this tile

    // ---- load: u with its halo, this thread's v, w, and D with its slopes ------------------------
    {
        const int nq4 = tq + 2, n = (th + 8) * nq4;
        for (int it = tid; it < n; it += nthr) {
            const int r = it / nq4 - 4, c = 4 * (it % nq4) - 4;
            const float *src = a.u + (int64_t)clampi(row0 + r, 0, H - 1) * pitch;
            float4 x;
            if (j0 + c >= 0 && j0 + c + 3 < W) {
                x = __ldcg(reinterpret_cast<const float4 *>(src + j0 + c));
            } else {
                x.x = __ldcg(src + clampi(j0 + c, 0, W - 1));
                x.y = __ldcg(src + clampi(j0 + c + 1, 0, W - 1));
                x.z = __ldcg(src + clampi(j0 + c + 2, 0, W - 1));
                x.w = __ldcg(src + clampi(j0 + c + 3, 0, W - 1));
            }
            st4(su + (r + UROW) * SUW + c + UCOL, x);
        }
    }
    // D the same into the second u buffer (free until the first step), for its slopes
    float *const sdt = su + SU;
    {
        const int nq4 = tq + 2, n = (th + 8) * nq4;
        for (int it = tid; it < n; it += nthr) {
            const int r = it / nq4 - 4, c = 4 * (it % nq4) - 4;
            const float *src = a.D + (int64_t)clampi(row0 + r, 0, H - 1) * pitch;
            float4 x;
            if (j0 + c >= 0 && j0 + c + 3 < W) {
                x = __ldg(reinterpret_cast<const float4 *>(src + j0 + c));
            } else {
                x.x = __ldg(src + clampi(j0 + c, 0, W - 1));
                x.y = __ldg(src + clampi(j0 + c + 1, 0, W - 1));
                x.z = __ldg(src + clampi(j0 + c + 2, 0, W - 1));
                x.w = __ldg(src + clampi(j0 + c + 3, 0, W - 1));
            }
            st4(sdt + (r + UROW) * SUW + c + UCOL, x);
        }
    }
    float4 v[R], w[R];
    if (mine) {
#pragma unroll
        for (int k = 0; k < R; ++k) {
            v[k] = w[k] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (k < k_lo) continue;
            // j is a multiple of 4 below W, and the pitch the next multiple of 4 at least
            v[k] = __ldcg(reinterpret_cast<const float4 *>(a.v + off0 + (int64_t)k * pitch));
            w[k] = __ldcg(reinterpret_cast<const float4 *>(a.w + off0 + (int64_t)k * pitch));
        }
    }
    __syncthreads();
    if (mine) {
#pragma unroll 1
        for (int x = 4 * k_lo; x < 4 * R; ++x) {
            const int k = x / 4, m = x % 4, i = i0 + k, jj = j + m < W ? j + m : W - 1;
            const float *p = sdt + (lr + k + UROW) * SUW + lc + m - (j + m - jj) + UCOL;
            float *d = reinterpret_cast<float *>(sD + k * nthr + tid) + m;
            d[0] = p[0];
            d[4 * R * nthr] = slope(p, SUW, i, H, rdx);
            d[8 * R * nthr] = slope(p, 1, jj, W, rdx);
        }
    }
    // the stimuli on during steps s .. s+31, one step per lane of warp 0
    auto fill_active = [&](int s) {
        const float t = (float)(ra.t0 + s + tid);
        unsigned on = 0;
        for (int q = 0; q < a.n_stim; ++q)
            if (stim_active(a.stim[q], t)) on |= 1u << q;
        s_active[(s & 32) + tid] = on;
    };
    if (tid < 32) fill_active(0);
    if (tid == 0) s_abort = 0;
    if (CL) {  // (the neighbours write into the second u buffer, which held D)
        cluster_arrive();
        cluster_wait();
    }
    __syncthreads();

    // strips: [0, 16 max_q) the tile's top 4 rows, then its bottom 4 rows, then its left and its
    // right 4 columns (4 words per row)
    const int64_t tile_g = blockIdx.x;
    const int o_bot = 16 * ra.max_q, o_left = 2 * o_bot, o_right = o_left + 4 * ra.max_g * R;
    const int n_top = tr > 0 ? 4 * tq : 0, n_bot = tr < t_nr - 1 ? 4 * tq : 0;
    const int n_left = tc > 0 ? th : 0, n_right = tc < t_nc - 1 ? th : 0;
    const int n_items = n_top + n_bot + n_left + n_right;
    // threads with a unit that meets a neighbour (whose cells it reads and sends): the block's first
    const int n_side = tq > 2 ? 2 * G + (gt + gb) * (tq - 2) : units;
    int n_ring = (n_side + 31) / 32 * 32;
    if (n_ring < n_items) n_ring = (n_items + 31) / 32 * 32;
    // Where few warps are at the sides, only they wait for the neighbours' strips (between two
    // barriers of their own) while the others go on; otherwise all wait, and one barrier is saved.
    const bool split = 4 * n_ring <= 3 * nthr;
    if (!split) n_ring = nthr;
    // item x of the strips this tile reads: where it lies (parity 0) and its place in a u buffer
    auto locate = [&](int x, const uint64_t *&src, int &dst) {
        int r, cc;
        int64_t t = tile_g, o;
        if (x < n_top) {  // the tile above: its bottom rows
            r = x / tq;
            cc = x - r * tq;
            r -= 4;
            t -= t_nc;
            o = o_bot + 4 * x;
        } else if ((x -= n_top) < n_bot) {  // the tile below: its top rows
            r = x / tq;
            cc = x - r * tq;
            r += th;
            t += t_nc;
            o = 4 * x;
        } else if ((x -= n_bot) < n_left) {
            r = x;
            cc = -1;
            t -= 1;
            o = o_right + 4 * x;
        } else {
            x -= n_left;
            r = x;
            cc = tq;
            t += 1;
            o = o_left + 4 * x;
        }
        src = ra.xchg + 2 * t * ra.slot + o;
        dst = (r + UROW) * SUW + 4 * cc + UCOL;
    };
    const uint64_t *in_src = ra.xchg;
    int in_dst = 0;
    if (tid < n_ring && tid < n_items) locate(tid, in_src, in_dst);
    // item x of the strips this tile sends (the same count): its place in a u buffer and in the
    // tile's strips
    auto locate_out = [&](int x, int &src, int &dst) {
        int r, cc;
        if (x < n_top) {
            r = x / tq;
            cc = x - r * tq;
            dst = 4 * x;
        } else if ((x -= n_top) < n_bot) {
            r = x / tq;
            cc = x - r * tq;
            r += th - 4;
            dst = o_bot + 4 * x;
        } else if ((x -= n_bot) < n_left) {
            r = x;
            cc = 0;
            dst = o_left + 4 * x;
        } else {
            r = x - n_left;
            cc = tq - 1;
            dst = o_right + 4 * r;
        }
        src = (r + UROW) * SUW + 4 * cc + UCOL;
    };
    int out_src = 0, out_dst = 0;
    if (tid < n_ring && tid < n_items) locate_out(tid, out_src, out_dst);
    // CL: item x's place in this tile's u buffer, and in its neighbour's (a shared::cluster address, buffer 0)
    auto locate_far = [&](int x, int &src, uint32_t &dst) {
        int r, cc, t, far_r, far_c;
        if (x < n_top) {  // the tile above: below its last row
            r = x / tq;
            cc = far_c = x - r * tq;
            t = tile - t_nc;
            far_r = row0 - (tr - 1) * t_ng / t_nr * R + r;
        } else if ((x -= n_top) < n_bot) {
            r = x / tq;
            cc = far_c = x - r * tq;
            t = tile + t_nc;
            far_r = r - 4;
            r += th - 4;
        } else if ((x -= n_bot) < n_left) {  // right of its last quad
            r = far_r = x;
            cc = 0;
            t = tile - 1;
            far_c = q0 - (tc - 1) * t_nq / t_nc;
        } else {
            r = far_r = x - n_left;
            cc = tq - 1;
            t = tile + 1;
            far_c = -1;
        }
        src = (r + UROW) * SUW + 4 * cc + UCOL;
        dst = cluster_addr(su + (far_r + UROW) * SUW + 4 * far_c + UCOL, t);
    };
    uint32_t far_dst = 0;
    if (CL && tid < n_items) locate_far(tid, out_src, far_dst);
    uint64_t *const out_strips = ra.xchg + 2 * tile_g * ra.slot;
    const int ucell = (lr + UROW) * SUW + lc + UCOL;
    auto any = [&](bool x) { return __any_sync(0xffffffffu, mine && x) != 0; };
    const Unit unit{i0, j, k_lo, off0, any(j == 0), any(j + 5 >= W - 1),
                    any(i0 <= (R == 2 ? 2 : 0)), any(i0 + R + (R == 2 ? 2 : 0) >= H)};
    int next_out = 0, next_step = ra.every ? 1 : ra.out_step[0];

    // a state that is written out
    auto write_out = [&](int s, const float *nxt) {
        if (s + 1 != next_step) return;
        const int64_t base = ra.every ? (int64_t)(s + 1) * ra.every : ra.out_off[next_out];
        float *const out = MANY && ra.base ? ra.base + tis.id * ra.tissue_stride : a.vo;
        const int64_t plane = (int64_t)H * pitch;
        ++next_out;
        next_step = ra.every ? s + 2 : next_out < ra.n_out ? ra.out_step[next_out] : 0;
        if (mine)
#pragma unroll
            for (int k = 0; k < R; ++k) {
                if (k < k_lo) continue;
                float *g = out + base + off0 + (int64_t)k * pitch;
                const float4 x = ld4(nxt + ucell + k * SUW);
                if (j + 3 < W) {
                    __stcg(reinterpret_cast<float4 *>(g), v[k]);
                    __stcg(reinterpret_cast<float4 *>(g + plane), w[k]);
                    __stcg(reinterpret_cast<float4 *>(g + 2 * plane), x);
                } else {
                    const float fv[4] = {v[k].x, v[k].y, v[k].z, v[k].w};
                    const float fw[4] = {w[k].x, w[k].y, w[k].z, w[k].w};
                    const float fu[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
                    for (int m = 0; m < 4; ++m)
                        if (j + m < W) {
                            __stcg(g + m, fv[m]);
                            __stcg(g + plane + m, fw[m]);
                            __stcg(g + 2 * plane + m, fu[m]);
                        }
                }
            }
    };

    for (int s = 0; s < ra.n; ++s) {
        const float *cur = su + (s & 1) * SU;
        float *nxt = su + ((s + 1) & 1) * SU;
        const bool last = s == ra.n - 1;
        const unsigned active = s_active[s & 63];
        const uint32_t tag = (uint32_t)s + 1;
        if (mine)
            step_unit<R, ACT>(a, tconst, kc, unit, cur + ucell, nxt + ucell, SUW, sD + tid, nthr, v, w,
                              active, (float)(ra.t0 + s));
        const int64_t par = (s & 1) * ra.slot;
        // Where the stores of a written state stand: of many tissues ahead of the barrier, where those of the warps
        // that are done overlap with the others' work (every state of 16 x 256^2: 9.7 us per step, behind the
        // strips 9.9); of one tissue behind the strips, out of the way of the code of a step that writes none
        // (1200^2 6.02 against 6.46 us, 1024^2 5.31 against 5.60, 128^2 1.83 against 1.89).
        if (MANY) write_out(s, nxt);
        if (!last) {
            if (tid < 32 && (s & 31) == 31) fill_active(s + 1);
            __syncthreads();
            // ---- this tile's strips out, and the neighbours' into the next buffer's halo ----------
            if (CL) {
                const uint32_t far_buf = ((s + 1) & 1) * SU * 4;
                for (int it = tid; it < n_items; it += nthr) {
                    if (it != tid) locate_far(it, out_src, far_dst);
                    st_cluster(far_dst + far_buf, ld4(nxt + out_src));
                }
                if (n_items > nthr && tid < n_items) locate_far(tid, out_src, far_dst);
                cluster_arrive();
            } else if (tid < n_ring) {
                for (int it = tid; it < n_items; it += n_ring) {
                    if (it != tid) locate_out(it, out_src, out_dst);
                    send_quad(out_strips + par + out_dst, ld4(nxt + out_src), tag);
                }
            }
        }
        if (!MANY) write_out(s, nxt);
        if (last) return;
        if (CL) {
            cluster_wait();
            continue;
        }
        if (tid < n_ring) {
            for (int it = tid; it < n_items; it += n_ring) {
                if (it != tid) locate(it, in_src, in_dst);
                float4 q;
                if (!wait_quad(in_src + par, tag, q)) {
                    s_abort = 1;
                    break;
                }
                st4(nxt + in_dst, q);
            }
            if (n_items > n_ring && tid < n_items) {  // more items than threads: back to the first
                locate_out(tid, out_src, out_dst);
                locate(tid, in_src, in_dst);
            }
            if (split) asm volatile("bar.sync 1, %0;" ::"r"(n_ring) : "memory");
        }
        if (!split) __syncthreads();
        // (split: the threads that do not wait see a wait that ran out after the next barrier at
        // the latest)
        if (s_abort) {
            if (tid == 0) atomicOr(a.status, kStatusTimeout);
            return;
        }
    }
}

// ---- plan and launch -----------------------------------------------------------------------------
// us per step, fitted to sweeps of (rows, tiles) over 64^2 .. 1200^2: the chain of one unit and the
// exchange, plus what the units sharing the SM add.
static double step_cost(int R, int units, int items) {
    static const double base[] = {0, 0, 2.0, 2.4, 3.3, 4.3};
    static const double each[] = {0, 0, 2.0e-3, 3.2e-3, 3.6e-3, 4.0e-3};
    return base[R] + each[R] * units + 5e-4 * items;
}

// The same with the tiles in one cluster: the faster one up to some 140^2 cells (us per step in a cluster | in
// blocks all over the device: 64^2 1.57 | 1.88, 128^2 1.62 | 1.88, 160^2 2.09 | 1.88, 200^2 2.31 | 1.97: 16 SMs
// have more units each).
static double cluster_cost(int units, int items) { return 1.66 + 2.0e-3 * units + 7e-4 * items; }

// Quads of a row of the u tile.  Of 8 lanes that load 16 bytes each, those beyond the end of a group of R rows
// go on in the next one: with this many quads in a row in the 16-byte banks after the others' (where R and the
// count allow it).  us per step without | with: 64^2 1.64 | 1.57, 128^2 1.76 | 1.62, 256^2 1.89 | 1.84, 1024^2
// 5.30 | 5.08, 1200^2 6.03 | 5.97 (27 % of the wavefronts there were conflicts).
static int tile_quads(int R, int max_q) {
    for (int x = max_q + 2; x < max_q + 10; ++x)
        if ((R * x - (max_q - 2)) % 8 == 0) return x;
    return max_q + 2;
}

// Every plan of at most `most` tiles with R rows per thread.
template <class F>
static void each_plan(int64_t H, int64_t W, int most, int R, F take) {
    if (H < 16 || W < 16 || most < 1 || H > 65536 || W > 65536 ||
        H * W > (int64_t)most * 512 * 4 * R)
        return;
    const int nq = (int)((W + 3) / 4);
    const int ng = (int)((H + R - 1) / R);
    // One tile row only where H is a multiple of R: with a shifted first group, row 0 and row H-1 must
    // lie in tiles of their own (see `shift`).
    for (int nr = ng * R == H ? 1 : 2; nr <= most && nr <= ng; ++nr) {
        // the smallest tile has ng / nr groups, the last one up to R - 1 rows less; strips take
        // 4 rows, a tile two quads (the last quad of the grid may be partial)
        if ((ng / nr) * R - (int)(ng * (int64_t)R - H) < 4) break;
        const int max_g = (ng + nr - 1) / nr;
        if (max_g > 512) continue;
        const int widest = 512 / max_g;  // quads of a tile: at most 512 units
        for (int nc = (nq + widest - 1) / widest; nc <= most / nr; ++nc) {
            if (nc > 1 && nq / nc < 2) break;
            const int max_q = (nq + nc - 1) / nc;
            const int units = max_g * max_q;
            const int items = (nr > 1 ? 8 * max_q : 0) + (nc > 1 ? 2 * max_g * R : 0);
            ResPlan p;
            p.rows = R;
            p.nr = nr;
            p.nc = nc;
            p.ng = ng;
            p.nq = nq;
            p.max_g = max_g;
            p.max_q = max_q;
            int want = units > items ? units : items;
            want = (want + 31) / 32 * 32;
            p.threads = want < 512 ? want : 512;
            p.su_h = max_g * R + 8 + R - 1;
            p.su_w = 4 * tile_quads(R, max_q);
            if (resident_smem(R, p.threads, p.su_w * p.su_h) > kResMaxSmem) p.su_w = 4 * (max_q + 2);
            p.smem = resident_smem(R, p.threads, p.su_w * p.su_h);
            if (p.smem > kResMaxSmem) continue;
            p.slot = 2 * 16 * (int64_t)max_q + 2 * 4 * (int64_t)max_g * R;
            p.tiles = nr * nc;
            p.cost = step_cost(R, units, items);
            take(p);
        }
    }
}

void resident_plans(int64_t H, int64_t W, int most, int R, std::vector<ResPlan> &best) {
    best.assign(most + 1, ResPlan());
    each_plan(H, W, most, R, [&](const ResPlan &p) {
        ResPlan &b = best[p.tiles];
        if (!b.ok() || p.cost < b.cost) b = p;
    });
    for (int t = 1; t <= most; ++t)
        if (!best[t].ok() || (best[t - 1].ok() && best[t - 1].cost <= best[t].cost)) best[t] = best[t - 1];
}

ResPlan resident_plan(int64_t H, int64_t W, int n_sm, int max_cluster) {
    ResPlan best;
    for (int R = kResMinRows; R <= kResMaxRows; ++R)
        each_plan(H, W, n_sm, R, [&](const ResPlan &p) {
            if (!best.ok() || p.cost < best.cost) best = p;
        });
    each_plan(H, W, max_cluster, kResClusterRows, [&](ResPlan p) {
        if (p.tiles & (p.tiles - 1)) return;
        p.cluster = true;
        p.cost = cluster_cost(p.max_g * p.max_q, (p.nr > 1 ? 8 * p.max_q : 0) + (p.nc > 1 ? 2 * p.max_g * p.rows : 0));
        if (p.cost < best.cost) best = p;
    });
    return best;
}

int resident_ctas() {
    static thread_local int dev_cached = -1, n_sm = 0;
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    if (dev != dev_cached) {
        int coop = 0;
        if (cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop)
            n_sm = 0;
        if (n_sm > kResMaxCtas) n_sm = kResMaxCtas;
        dev_cached = dev;
    }
    return n_sm;
}

template <int R, bool ACT, bool MANY, bool CL>
static cudaError_t configure() {
    // the attributes are per function and per context: set again whenever the context changes
    static thread_local uint64_t configured_ctx = 0;
    if (!context_changed(configured_ctx)) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(fk_resident_kernel<R, ACT, MANY, CL>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kResMaxSmem);
    if (CL && e == cudaSuccess)
        e = cudaFuncSetAttribute(fk_resident_kernel<R, ACT, MANY, CL>, cudaFuncAttributeNonPortableClusterSizeAllowed,
                                 1);
    if (e != cudaSuccess) configured_ctx = 0;
    return e;
}

// Launch of `ctas` blocks that run at the same time: cooperative, or one cluster.
struct ResLaunch {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    ResLaunch(int ctas, int threads, size_t smem, bool cluster, cudaStream_t stream) {
        cfg.gridDim = dim3((unsigned)ctas);
        cfg.blockDim = dim3((unsigned)threads);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = stream;
        if (cluster) {
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = (unsigned)ctas;
            attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        } else {
            attr[0].id = cudaLaunchAttributeCooperative;
            attr[0].val.cooperative = 1;
        }
        cfg.attrs = attr;
        cfg.numAttrs = 1;
    }
};

// The largest cluster (16, 8 or none: 0) of full-size blocks that the current device takes.
static int resident_cluster() {
    static thread_local int dev_cached = -1, most = 0;
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    if (dev != dev_cached) {
        most = 0;
        if (resident_ctas() > 0 && configure<kResClusterRows, false, false, true>() == cudaSuccess)
            for (int c = 16; c >= 8 && most == 0; c /= 2) {
                ResLaunch l(c, 512, kResMaxSmem, true, nullptr);
                int n = 0;
                if (cudaOccupancyMaxActiveClusters(&n, fk_resident_kernel<kResClusterRows, false, false, true>,
                                                   &l.cfg) == cudaSuccess && n >= 1)
                    most = c;
                else
                    cudaGetLastError();
            }
        dev_cached = dev;
    }
    return most;
}

ResPlan resident_plan(int64_t H, int64_t W) { return resident_plan(H, W, resident_ctas(), resident_cluster()); }

template <int R, bool ACT, bool MANY, bool CL = false>
static cudaError_t launch_one(const cudaLaunchConfig_t &cfg, const ResidentArgs &ra, const StepArgs &a,
                              const PackConsts &k) {
    const cudaError_t e = configure<R, ACT, MANY, CL>();
    return e != cudaSuccess ? e : cudaLaunchKernelEx(&cfg, fk_resident_kernel<R, ACT, MANY, CL>, ra, a, k);
}
template <int R>
static cudaError_t launch_rows(const cudaLaunchConfig_t &cfg, const ResidentArgs &ra, const StepArgs &a,
                               const PackConsts &k) {
    if (ra.tissues) return launch_one<R, false, true>(cfg, ra, a, k);
    return a.act_last ? launch_one<R, true, false>(cfg, ra, a, k) : launch_one<R, false, false>(cfg, ra, a, k);
}

static cudaError_t launch_any(int rows, int ctas, int threads, size_t smem, bool cluster, const ResidentArgs &ra,
                              const StepArgs &a, cudaStream_t stream) {
    const ResLaunch l(ctas, threads, smem, cluster, stream);
    const PackConsts k = make_pack_consts(a.m, a.rdx, a.dt);
    if (cluster) {
        if (rows != kResClusterRows || ra.tissues) return cudaErrorInvalidValue;
        return a.act_last ? launch_one<kResClusterRows, true, false, true>(l.cfg, ra, a, k)
                          : launch_one<kResClusterRows, false, false, true>(l.cfg, ra, a, k);
    }
    switch (rows) {
        case 2: return launch_rows<2>(l.cfg, ra, a, k);
        case 3: return launch_rows<3>(l.cfg, ra, a, k);
        case 4: return launch_rows<4>(l.cfg, ra, a, k);
        case 5: return launch_rows<5>(l.cfg, ra, a, k);
        default: return cudaErrorInvalidValue;
    }
}

static thread_local int refusals = 0;
void refuse_resident_launches(int n) { refusals = n; }

cudaError_t launch_resident(int rows, int ctas, int threads, size_t smem, bool cluster, const ResidentArgs &ra,
                            const StepArgs &a, cudaStream_t stream) {
    if (refusals > 0) {
        --refusals;
        return kResRefused;
    }
    const cudaError_t e = launch_any(rows, ctas, threads, smem, cluster, ra, a, stream);
    switch (e) {
        case cudaErrorCooperativeLaunchTooLarge:
        case cudaErrorInvalidClusterSize:
        case cudaErrorLaunchOutOfResources:
            cudaGetLastError();  // (not the next call's error)
            return kResRefused;
        default: return e;
    }
}

}  // namespace fk
