// Adjoint of the marker step with respect to the initial marker temperatures and
// the amplitudes of velocity modes, v = sum_m a_m (vx_m, vy_m).
//
// Forward model (what i2g_adjoint_forward runs): nsteps x {movemark; ronurecalc}
// with the combined velocity field, positions checkpointed (by caller index)
// every k steps.  Loss gradient dL/dtk is given at the final node temperatures
// tk = sum_i w_i T_i / sum_i w_i (markmart.c:899-906, 988-991).
//
// Reverse:
//   k_adj_avg   per marker: dL/dT_i = sum_n g_n w_in / W_n and
//               dL/dx_i = sum_n g_n (T_i - tk_n) / W_n dw_in/dx_i over its 2x2
//               nodes; temperatures the step replaced (sticky air, out of box)
//               get zero.
//   k_adj_rk4   per marker, independent of every other marker: for each
//               checkpoint segment, last first, recompute the segment's positions
//               with the forward's own arithmetic, then run the reverse of the
//               classical RK4 stage chain, using the bilinear Jacobian of the
//               velocity at every stage point and the mode velocities for
//               dL/da; per-CTA partial sums of dL/da, folded in a fixed order.
// The interpolants are piecewise bilinear; derivatives are those of the piece
// the forward used (the stencil switches at faces and midpoints have measure zero).
#pragma once

#include "i2g_kernels.cuh"

namespace i2g {

constexpr int kMaxModes = 16;
constexpr int kMaxCkptSeg = 16;  // steps per checkpoint segment held in registers

struct AdjView {
    // [nn][capacity] unit-amplitude mode velocities, interleaved, zero beyond the
    // modes set; the capacity is 4, 8 or 16 (mode_capacity), so a node's modes are
    // whole 16-byte loads
    const double *mvx, *mvy;
};

__host__ __device__ constexpr int mode_capacity(int nmodes) { return nmodes <= 4 ? 4 : (nmodes <= 8 ? 8 : 16); }

// The stencils of allinterv() at a point: vx on basic columns and staggered rows
// at lower node (ax, ay), vy on staggered columns and basic rows at (bx, by), with
// the upper (1) and lower (0) weights of each axis.  inx, iny: the point was not
// clamped to the box along that axis (clamped: no dependence on it).
template <bool MIXED>
struct __align__(16) VStencil {
    int ax, ay, bx, by;  // ax, ay negative (complemented): clamped along x, y
    double xa0, xa1, ya0, ya1, xb0, xb1, yb0, yb1;
};
// the mixed form: FP32 upper weights; a lower weight is 1 - upper, as AxisF has it
template <>
struct __align__(16) VStencil<true> {
    int ax, ay, bx, by;
    float xa1, ya1, xb1, yb1;
};
static_assert(sizeof(VStencil<true>) == 32 && sizeof(VStencil<false>) == 80, "whole 16-byte pieces");
template <bool MIXED>
__device__ __forceinline__ void a_weights(const VStencil<MIXED> &S, double (&x)[2], double (&y)[2])
{
    if constexpr (MIXED) {
        x[0] = (double)(1.0f - S.xa1); x[1] = (double)S.xa1; y[0] = (double)(1.0f - S.ya1); y[1] = (double)S.ya1;
    } else {
        x[0] = S.xa0; x[1] = S.xa1; y[0] = S.ya0; y[1] = S.ya1;
    }
}
template <bool MIXED>
__device__ __forceinline__ void b_weights(const VStencil<MIXED> &S, double (&x)[2], double (&y)[2])
{
    if constexpr (MIXED) {
        x[0] = (double)(1.0f - S.xb1); x[1] = (double)S.xb1; y[0] = (double)(1.0f - S.yb1); y[1] = (double)S.yb1;
    } else {
        x[0] = S.xb0; x[1] = S.xb1; y[0] = S.yb0; y[1] = S.yb1;
    }
}

// hx, hy: a nearby cell to start the searches from (-1: none), replaced by the point's
template <bool MIXED>
__device__ __forceinline__ VStencil<MIXED> v_stencil(const GridView &G, double x, double y, int &hx, int &hy)
{
    VStencil<MIXED> S;
    const double xc = x, yc = y;
    clampxy(G, x, y);
    if constexpr (MIXED) {
        AxisF X, Y;
        axis_fast(G.gx, G.lx, G.nx, G.inv_x, x, hx, X);
        axis_fast(G.gy, G.ly, G.ny, G.inv_y, y, hy, Y);
        hx = X.b;
        hy = Y.b;
        S.ax = X.b; S.ay = Y.m; S.bx = X.m; S.by = Y.b;
        S.xa1 = X.b1; S.ya1 = Y.m1; S.xb1 = X.m1; S.yb1 = Y.b1;
    } else {
        const int nx = (int)G.nx, ny = (int)G.ny;
        const int m10 = hx >= 0 ? cell_walk(G.gx, nx, hx, x) : (int)cell_search(G.gx, G.nx, G.inv_x, x);
        const int m20 = hy >= 0 ? cell_walk(G.gy, ny, hy, y) : (int)cell_search(G.gy, G.ny, G.inv_y, y);
        hx = m10;
        hy = m20;
        int m2 = m20, m1 = m10;
        if (y < __ldg(G.ymid + m20)) m2 -= 1;
        m2 = min(max(m2, 0), ny - 3);
        if (x < __ldg(G.xmid + m10)) m1 -= 1;
        m1 = min(max(m1, 0), nx - 3);
        S.ax = m10; S.ay = m2; S.bx = m1; S.by = m20;
        fdw64(__ldg(G.gx + m10), __ldg(G.gx + m10 + 1), x, S.xa0, S.xa1);
        fdw64(__ldg(G.ymid + m2), __ldg(G.ymid + m2 + 1), y, S.ya0, S.ya1);
        fdw64(__ldg(G.xmid + m1), __ldg(G.xmid + m1 + 1), x, S.xb0, S.xb1);
        fdw64(__ldg(G.gy + m20), __ldg(G.gy + m20 + 1), y, S.yb0, S.yb1);
    }
    if (x != xc) S.ax = ~S.ax;
    if (y != yc) S.ay = ~S.ay;
    return S;
}

__device__ __forceinline__ int unclamped(int a) { return a < 0 ? ~a : a; }

// the velocity from a point's stencils, with the forward's arithmetic
template <bool MIXED>
__device__ __forceinline__ void v_value(const GridView &G, const VStencil<MIXED> &S, double &vx, double &vy)
{
    const int ax = unclamped(S.ax), ay = unclamped(S.ay);
    if constexpr (MIXED) {
        vx = (double)bil32i(G.vxf, (int)G.ny, ax, ay, 1.0f - S.xa1, S.xa1, 1.0f - S.ya1, S.ya1);
        vy = (double)bil32i(G.vyf, (int)G.ny, S.bx, S.by, 1.0f - S.xb1, S.xb1, 1.0f - S.yb1, S.yb1);
    } else {
        vx = bil64(G.vx, G.ny, ax, ay, S.xa0, S.xa1, S.ya0, S.ya1);
        vy = bil64(G.vy, G.ny, S.bx, S.by, S.xb0, S.xb1, S.yb0, S.yb1);
    }
}

// (kx, ky) times the velocity's Jacobian at a point: dL/dx of the stage
template <bool MIXED>
__device__ __forceinline__ void v_pull(const GridView &G, const VStencil<MIXED> &S, double kx, double ky, double &px,
                                       double &py)
{
    const int ny = (int)G.ny, ax = unclamped(S.ax), ay = unclamped(S.ay);
    double dxa, dya, dxb, dyb;  // d(w1)/dx, d(w1)/dy of the vx and the vy stencil
    if constexpr (MIXED) {
        dxa = __ldg(G.lx + ax).y;
        dya = __ldg(G.ly + ay).z;
        dxb = __ldg(G.lx + S.bx).z;
        dyb = __ldg(G.ly + S.by).y;
    } else {
        dxa = 1.0 / (__ldg(G.gx + ax + 1) - __ldg(G.gx + ax));
        dya = 1.0 / (__ldg(G.ymid + ay + 1) - __ldg(G.ymid + ay));
        dxb = 1.0 / (__ldg(G.xmid + S.bx + 1) - __ldg(G.xmid + S.bx));
        dyb = 1.0 / (__ldg(G.gy + S.by + 1) - __ldg(G.gy + S.by));
    }
    // corner values: the FP64 grids in both forms
    const double *pa = G.vx + (int64_t)ax * ny + ay, *pb = G.vy + (int64_t)S.bx * ny + S.by;
    const double a00 = __ldg(pa), a01 = __ldg(pa + 1), a10 = __ldg(pa + ny), a11 = __ldg(pa + ny + 1);
    const double b00 = __ldg(pb), b01 = __ldg(pb + 1), b10 = __ldg(pb + ny), b11 = __ldg(pb + ny + 1);
    double xa[2], ya[2], xb[2], yb[2];
    a_weights<MIXED>(S, xa, ya);
    b_weights<MIXED>(S, xb, yb);
    const double dx = kx * (dxa * (ya[0] * (a10 - a00) + ya[1] * (a11 - a01))) +
                      ky * (dxb * (yb[0] * (b10 - b00) + yb[1] * (b11 - b01)));
    const double dy = kx * (dya * (xa[0] * (a01 - a00) + xa[1] * (a11 - a10))) +
                      ky * (dyb * (xb[0] * (b01 - b00) + xb[1] * (b11 - b10)));
    px = S.ax >= 0 ? dx : 0.0;
    py = S.ay >= 0 ? dy : 0.0;
}

// dL/da of one velocity component.  A stage adds k x (corner weight) x (mode
// velocity at the corner) to every mode.  Along a marker's path many stages in a
// row use the same stencil, so their corner weights are summed first and meet the
// modes once per stencil.
template <int NM>
struct ModeRun {
    int64_t node;  // lower node of the open stencil, -1: none
    double w[4];
    __device__ __forceinline__ void open()
    {
        node = -1;
        w[0] = w[1] = w[2] = w[3] = 0.0;
    }
    __device__ __forceinline__ void close(const double *__restrict__ mv, int ny, double (&da)[NM])
    {
        const double2 *p = reinterpret_cast<const double2 *>(mv + node * NM);
        const int up = ny * (NM / 2);
#pragma unroll
        for (int h = 0; h < NM / 2; h++) {
            const double2 q0 = __ldg(p + h), q1 = __ldg(p + NM / 2 + h), q2 = __ldg(p + up + h),
                          q3 = __ldg(p + up + NM / 2 + h);
            da[2 * h] += w[0] * q0.x + w[1] * q1.x + w[2] * q2.x + w[3] * q3.x;
            da[2 * h + 1] += w[0] * q0.y + w[1] * q1.y + w[2] * q2.y + w[3] * q3.y;
        }
    }
    __device__ __forceinline__ void add(const double *__restrict__ mv, int ny, int64_t at, double k,
                                        const double (&x)[2], const double (&y)[2], double (&da)[NM])
    {
        if (at != node) {
            if (node >= 0) close(mv, ny, da);
            node = at;
            w[0] = w[1] = w[2] = w[3] = 0.0;
        }
        const double k0 = k * x[0], k1 = k * x[1];
        w[0] += k0 * y[0];
        w[1] += k0 * y[1];
        w[2] += k1 * y[0];
        w[3] += k1 * y[1];
    }
};

// one forward step of a marker exactly as movemark() moves it (velocity only)
template <bool MIXED>
__device__ __forceinline__ void rk4_forward(const GridView &G, const MoveArgs &A, double &x, double &y)
{
    double vx0, vy0;
    const double dt = A.timestep;
    if (MIXED) {
        int hx, hy;
        rk4_mixed(G, x, y, dt, A.markmod, vx0, vy0, nullptr, hx, hy);
    } else {
        if (A.markmod == 1) {
            interp_v<false>(G, x, y, vx0, vy0);
        } else {
            double vx1, vy1, vx2, vy2, vx3, vy3, vx4, vy4;
            interp_v<false>(G, x, y, vx1, vy1);
            interp_v<false>(G, x + vx1 * dt / 2.0, y + vy1 * dt / 2.0, vx2, vy2);
            interp_v<false>(G, x + vx2 * dt / 2.0, y + vy2 * dt / 2.0, vx3, vy3);
            interp_v<false>(G, x + vx3 * dt, y + vy3 * dt, vx4, vy4);
            vx0 = (vx1 + 2.0 * vx2 + 2.0 * vx3 + vx4) / 6.0;
            vy0 = (vy1 + 2.0 * vy2 + 2.0 * vy3 + vy4) / 6.0;
        }
    }
    if (A.outgrid == 2) {
        if (x < 0 || x > G.xsize) vy0 = 0;
        if (y < 0 || y > G.ysize) vx0 = 0;
    }
    x += dt * vx0;
    y += dt * vy0;
}

constexpr int kAdjThreads = 128;

// a thread's stencils of the four stages, 16 bytes of every thread side by side
template <bool MIXED>
struct StageStore {
    static constexpr int NP = sizeof(VStencil<MIXED>) / 16;
    uint4 q[4][NP][kAdjThreads];
    __device__ __forceinline__ void put(int st, const VStencil<MIXED> &S)
    {
        const uint4 *u = reinterpret_cast<const uint4 *>(&S);
#pragma unroll
        for (int k = 0; k < NP; k++) q[st][k][threadIdx.x] = u[k];
    }
    __device__ __forceinline__ VStencil<MIXED> get(int st) const
    {
        VStencil<MIXED> S;
        uint4 *u = reinterpret_cast<uint4 *>(&S);
#pragma unroll
        for (int k = 0; k < NP; k++) u[k] = q[st][k][threadIdx.x];
        return S;
    }
};

// reverse of one step from (x, y): lam (dL/dx after the step) -> dL/dx before it,
// the stages' dL/da into the open runs.  The stencils of the stages are found once,
// on the way to the fourth stage point, and kept in shared memory; both passes are
// loops over the stages, which keeps the kernel's code within the instruction
// cache (unrolled: 1.76 ms, the loops: 1.47).
template <bool MIXED, int NM>
__device__ __forceinline__ void rk4_reverse(const GridView &G, const AdjView &Md, const MoveArgs &A,
                                            StageStore<MIXED> &Q, double x, double y, int &hx, int &hy, double &lx,
                                            double &ly, ModeRun<NM> &rx, ModeRun<NM> &ry, double (&da)[NM])
{
    const double dt = A.timestep;
    const int ny = (int)G.ny, nst = A.markmod == 1 ? 1 : 4;
    double ox = 1.0, oy = 1.0;  // orthogonal-only motion outside the box (markmart.c:100-105)
    if (A.outgrid == 2) {
        if (x < 0 || x > G.xsize) oy = 0.0;
        if (y < 0 || y > G.ysize) ox = 0.0;
    }
    // dL/d(vx0, vy0) of x' = x + dt*v0
    const double g0x = lx * dt * ox, g0y = ly * dt * oy;
    // stage points (recomputed with the forward's arithmetic): x, then x + v dt / 2
    // twice, then x + v dt
    double qx = x, qy = y;
#pragma unroll 1
    for (int st = 0; st < nst; st++) {
        const VStencil<MIXED> S = v_stencil<MIXED>(G, qx, qy, hx, hy);
        Q.put(st, S);
        if (st + 1 < nst) {
            double vx, vy;
            v_value<MIXED>(G, S, vx, vy);
            const double h = st == 2 ? dt : 0.5 * dt;
            qx = x + vx * h;
            qy = y + vy * h;
        }
    }
    // v0 = (v1 + 2 v2 + 2 v3 + v4) / 6; a stage point's own dependence on the stage
    // before it enters that stage's factor
    double px = 0.0, py = 0.0;
    const double ax = nst == 1 ? g0x : sixth_of(g0x), ay = nst == 1 ? g0y : sixth_of(g0y);
#pragma unroll 1
    for (int st = nst - 1; st >= 0; st--) {
        const double c = st == 0 || st == 3 ? 1.0 : 2.0;
        const double h = st == 2 ? dt : 0.5 * dt;  // (the last stage: px = py = 0)
        const double kx = ax * c + h * px, ky = ay * c + h * py;
        const VStencil<MIXED> S = Q.get(st);
        double wx[2], wy[2];
        a_weights<MIXED>(S, wx, wy);
        rx.add(Md.mvx, ny, (int64_t)unclamped(S.ax) * ny + unclamped(S.ay), kx, wx, wy, da);
        b_weights<MIXED>(S, wx, wy);
        ry.add(Md.mvy, ny, (int64_t)S.bx * ny + S.by, ky, wx, wy, da);
        v_pull<MIXED>(G, S, kx, ky, px, py);
        lx += px;
        ly += py;
    }
}

// averaging adjoint at the final positions (device order); outputs by caller index
template <bool MIXED>
__global__ void __launch_bounds__(256) k_adj_avg(const __grid_constant__ GridView G,
                                                 const __grid_constant__ MarkerView M, const DevTypes *__restrict__ Ty,
                                                 int32_t gridmod, double tmp_ambient, const double *__restrict__ tk,
                                                 const double *__restrict__ w1, const double *__restrict__ g,
                                                 const double *__restrict__ T0, double2 *__restrict__ lam,
                                                 double *__restrict__ dT)
{
    const i2g_types &T = Ty->t;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    const int64_t ny = G.ny;
    for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < M.n; j += stride) {
        const int32_t id = M.id[j];
        const double x = M.x[j], y = M.y[j], Tm = M.T[j];
        const int mt = M.type[j];
        double gT = 0.0, gx = 0.0, gy = 0.0;
        const bool valid = x > 0 && y > 0 && x < G.xsize && y < G.ysize && Tm > 0 && mt < 50 &&
                           (gridmod <= 1 || (id % gridmod) == 0) && !T.markim[mt];
        if (valid) {
            const int64_t m10 = cell_search(G.gx, G.nx, G.inv_x, x), m20 = cell_search(G.gy, ny, G.inv_y, y);
            double wx0, wx1, wy0, wy1, ix, iy;
            if (!MIXED) {
                fdw64(__ldg(G.gx + m10), __ldg(G.gx + m10 + 1), x, wx0, wx1);
                fdw64(__ldg(G.gy + m20), __ldg(G.gy + m20 + 1), y, wy0, wy1);
                ix = 1.0 / (__ldg(G.gx + m10 + 1) - __ldg(G.gx + m10));
                iy = 1.0 / (__ldg(G.gy + m20 + 1) - __ldg(G.gy + m20));
            } else {
                float a0, a1, b0, b1;
                fdw32(__ldg(G.gx + m10), __ldg(G.ixb + m10), x, a0, a1);
                fdw32(__ldg(G.gy + m20), __ldg(G.iyb + m20), y, b0, b1);
                wx0 = a0; wx1 = a1; wy0 = b0; wy1 = b1;
                ix = __ldg(G.ixb + m10);
                iy = __ldg(G.iyb + m20);
            }
            const double wx[2] = {wx0, wx1}, wy[2] = {wy0, wy1}, dwx[2] = {-ix, ix}, dwy[2] = {-iy, iy};
            for (int a = 0; a < 2; a++)
                for (int b = 0; b < 2; b++) {
                    const int64_t m3 = (m10 + a) * ny + m20 + b;
                    const double W = w1[m3];
                    if (!(W > 0)) continue;
                    const double c = g[m3] / W, r = Tm - tk[m3];
                    gT += c * wx[a] * wy[b];
                    gx += c * r * dwx[a] * wy[b];
                    gy += c * r * wx[a] * dwy[b];
                }
        }
        // temperatures replaced by the step (sticky air, out of the box) carry no gradient
        const bool replaced = mt < 2 || Tm != T0[id];
        dT[id] = replaced ? 0.0 : gT;
        lam[id] = make_double2(gx, gy);
    }
}

// Reverse through all steps, one thread per marker (caller index).  Bound by the
// latency and the FP64 rate of the stage chain; every array the steps index is in
// registers (the mode count is a template parameter) except the segment's
// positions and the stage stencils (shared memory).  640k markers, 20 steps, 8
// modes, mixed: 5.55 ms with run-time mode loops (their arrays in local memory) and
// every stage meeting every mode, 2.71 with ModeRun and the modes in registers, 1.47
// with the stages as loops and five CTAs per SM (four: 1.50, six: 1.73, spills).
template <bool MIXED, int NM>
__global__ void __launch_bounds__(kAdjThreads, MIXED && NM <= 8 ? 5 : 3) k_adj_rk4(const __grid_constant__ GridView G,
                                                 const __grid_constant__ AdjView Md,
                                                 const __grid_constant__ MoveArgs A, const DevTypes *__restrict__ Ty,
                                                 const int8_t *__restrict__ type_by_id, const double2 *__restrict__ ck,
                                                 int64_t n, int32_t nsteps, int32_t every, double2 *__restrict__ lam,
                                                 double *__restrict__ dapart, int32_t nm)
{
    __shared__ __align__(16) union Smem {
        StageStore<MIXED> Q;
        double red[NM][kAdjThreads];
        __device__ Smem() {}
    } S;
    const i2g_types &T = Ty->t;
    double da[NM];
#pragma unroll
    for (int m = 0; m < NM; m++) da[m] = 0.0;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        double2 l = lam[i];
        double lx = l.x, ly = l.y;
        const bool moves = !T.markim[type_by_id[i]];
        const int nseg = (nsteps + every - 1) / every;
        ModeRun<NM> rx, ry;
        rx.open();
        ry.open();
        int hx = -1, hy = -1;
        for (int sg = nseg - 1; sg >= 0; sg--) {
            const int s0 = sg * every, len = min(every, nsteps - s0);
            double xs[kMaxCkptSeg], ys[kMaxCkptSeg];
            double2 p = ck[(int64_t)sg * n + i];
            double x = p.x, y = p.y;
            for (int s = 0; s < len; s++) {
                xs[s] = x;
                ys[s] = y;
                if (s + 1 == len) break;  // the segment's last step is not needed again
                const bool inbox = (x >= 0 && y >= 0 && x <= G.xsize && y <= G.ysize);
                if ((inbox || A.outgrid != 1) && moves) rk4_forward<MIXED>(G, A, x, y);
            }
            for (int s = len - 1; s >= 0; s--) {
                const double xx = xs[s], yy = ys[s];
                const bool inbox = (xx >= 0 && yy >= 0 && xx <= G.xsize && yy <= G.ysize);
                if ((inbox || A.outgrid != 1) && moves)
                    rk4_reverse<MIXED, NM>(G, Md, A, S.Q, xx, yy, hx, hy, lx, ly, rx, ry, da);
            }
        }
        if (rx.node >= 0) rx.close(Md.mvx, (int)G.ny, da);
        if (ry.node >= 0) ry.close(Md.mvy, (int)G.ny, da);
        lam[i] = make_double2(lx, ly);
    }
    // per-CTA partial sums of dL/da (fixed tree order: deterministic)
    __syncthreads();  // the stage stores are done
#pragma unroll
    for (int m = 0; m < NM; m++) S.red[m][threadIdx.x] = da[m];
    __syncthreads();
    for (int s = kAdjThreads / 2; s > 0; s >>= 1) {
        if ((int)threadIdx.x < s)
#pragma unroll
            for (int m = 0; m < NM; m++) S.red[m][threadIdx.x] += S.red[m][threadIdx.x + s];
        __syncthreads();
    }
    if ((int)threadIdx.x < nm) dapart[(int64_t)blockIdx.x * nm + threadIdx.x] = S.red[threadIdx.x][0];
}

template <bool MIXED>
static void launch_adj_rk4(cudaStream_t s, const GridView &G, const AdjView &Md, const MoveArgs &A,
                           const DevTypes *types, int64_t n, int32_t nm, const int8_t *type_by_id, const double2 *ck,
                           int32_t nsteps, int32_t every, double2 *lam, double *dapart, int32_t nblk)
{
    switch (mode_capacity(nm)) {
    case 4:
        k_adj_rk4<MIXED, 4><<<nblk, kAdjThreads, 0, s>>>(G, Md, A, types, type_by_id, ck, n, nsteps, every, lam, dapart,
                                                         nm);
        break;
    case 8:
        k_adj_rk4<MIXED, 8><<<nblk, kAdjThreads, 0, s>>>(G, Md, A, types, type_by_id, ck, n, nsteps, every, lam, dapart,
                                                         nm);
        break;
    default:
        k_adj_rk4<MIXED, 16><<<nblk, kAdjThreads, 0, s>>>(G, Md, A, types, type_by_id, ck, n, nsteps, every, lam,
                                                          dapart, nm);
    }
}

}  // namespace i2g
