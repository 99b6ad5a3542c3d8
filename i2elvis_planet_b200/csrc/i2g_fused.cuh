// The mixed-precision marker step in two passes over memory: movemark() with the
// marker's averaging contribution (markmart.c:23-155 then the marker loop of
// markmart.c:271-913), and the per-cell sums with the node loop
// (markmart.c:917-993) in one kernel.
//
//   k_move_fused   persistent CTAs over tiles of 256 markers in storage order,
//                  the next tile's fields staged in shared memory: RK4 through
//                  the staggered grid (on a uniform grid from arithmetic and the
//                  per-quarter-cell velocity forms, no line tables), the new
//                  position and pressure, then the marker's 16-byte averaging
//                  record at its new cell: fixed-point weights, temperature, the
//                  type's slot, and the log-viscosity in the spare bits.  The
//                  record goes to the next free place of its cell's bucket
//                  (ncells x cap places; a full bucket spills to an overflow
//                  list).  No sort: the markers stay where they are.
//   k_cellnodes    a CTA per tile of 31 x (8G - 1) nodes: a warp per cell column,
//                  a lane per cell (two on small grids), each lane adds its cell's
//                  records into per-slot sums; the cells' sums meet in shared
//                  memory, where a thread per node finishes it.
//
// Order independence.  The records arrive in their buckets in whatever order the
// atomics grant, so every sum is made exact, and exact sums do not depend on the
// order of their terms:
//   - every term of a sum (corner, quadrant and cell-centre weights, temperature
//     x weight, log-viscosity x weight) is rounded to a quantum q of its own sum,
//     a power of two fixed per call by the largest |term| and the largest cell
//     count, after which its FP64 sums are exact;
//   - density, heat capacity, conductivity and heat depend on the rock type alone
//     on these calls, so their sums are per-type weight sums (exact) times the
//     type's values, combined in a fixed order.
// The node values are therefore bitwise the same for every run, launch shape and
// marker storage order.  A node whose temperature or viscosity weight sum is so
// small that the quantum would cost more than 1e-9 of the value is recomputed by
// node_guard with quanta of its own.
#pragma once

#include "i2g_avg.cuh"

namespace i2g {

// ----------------------------------------------------------------- layout
constexpr int kFusedParts = 64;  // per-block statistics are spread over this many slots

struct FusedCounters {
    // per slot (block index mod kFusedParts): largest cell count, largest |tk|
    // and |log-viscosity| (FP32 bit patterns of upper bounds), averaged markers
    uint32_t part[kFusedParts][4];
    int32_t novf, ntreset;  // overflow records, pending sticky-air resets
    int32_t ndefer;         // records whose log-viscosity k_fused_begin writes
    int32_t any;            // any node viscosity written
    unsigned long long kmin, kmax;  // ordered keys of the smallest / largest node viscosity
};

struct OvfRec {
    float4 a;  // the record (rec_pack)
    int32_t cell, pad[3];
};

struct FusedMove {
    AvgArgsK avg;                // the averaging's constants
    uint8_t type[kAvgTypes];     // per rock type: rec_type_byte
    int32_t cap;                 // places per bucket
    float4 *ra;                  // [cells, whole strips of 32, * cap] the records (rec_pack, rec_place)
    OvfRec *ovf;                 // [markers]
    int32_t *count;              // [ncells] records per cell (zeroed before the launch)
    FusedCounters *ctr;          // zeroed before the launch
    int32_t *spilled;            // host memory: set to 1 by a call that overflows a bucket
    int32_t *treset;             // [markers] markers whose T the averaging resets
    int2 *defer;                 // [markers] {marker, record place} of markers without a viscosity
    // a step replayed from a CUDA graph: the step's timesum from a device table
    // (stepc[4 * *stepi]) instead of avg.timesum; NULL otherwise
    const double *stepc;
    const int32_t *stepi;
};

// ----------------------------------------------------------------- uniform axes
// Floors and small int -> float/double casts without conversion instructions
// (which share the SM's narrow XU pipe with log2f and the FP32/FP64 casts):
// adding 2^52 to an FP64 t in [-2^51, 2^51] with rounding down leaves
// 2^52 + floor(t), whose low word is floor(t); adding 1.5 x 2^23 to an FP32 u
// with |u| < 2^22 rounding down leaves a number whose bit pattern counts units
// from 1.5 x 2^23.  The results equal __double2int_rd, __float2int_rd and the
// casts exactly.
constexpr float kF32Magic = 12582912.0f;  // 1.5 x 2^23, bit pattern 0x4B400000
__device__ __forceinline__ int floor_dm(double t) { return __double2loint(__dadd_rd(t, 0x1p52)); }
__device__ __forceinline__ double dbl_of(int k) { return __hiloint2double(0x43300000, k) - 0x1p52; }  // k >= 0
__device__ __forceinline__ int floor_fm(float u, float &fl)
{
    const float s = __fadd_rd(u, kF32Magic);
    fl = s - kF32Magic;
    return __float_as_int(s) - 0x4B400000;
}
__device__ __forceinline__ float flt_of(int d) { return __int_as_float(0x4B400000 + d) - kF32Magic; }  // |d| < 2^22
// max and min that pass a NaN on, as "if (e < lo) e = lo" does, in one instruction
__device__ __forceinline__ float max_nan(float a, float b)
{
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float min_nan(float a, float b)
{
    float r;
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
// The stencil choice and weights of one axis (AxisF) on a uniform axis: b1 is the
// coordinate inside basic cell b in cells; the staggered stencil is the lower or
// upper neighbour by the half-cell, clamped to [0, n-3], with its weight
// (markmart.c:1403-1409, 1431-1437, 1514-1520).
__device__ __forceinline__ void uni_tail(int n, int b, float b1, AxisF &A)
{
    A.b = b;
    A.b1 = b1;
    A.b0 = 1.0f - b1;
    int m = (b1 < 0.5f) ? b - 1 : b;
    if (m < 0) m = 0;
    if (m > n - 3) m = n - 3;
    const float t = b1 - 0.5f + (m != b ? 1.0f : 0.0f);  // (float)(b - m): 0 or 1
    A.m = m;
    A.m1 = t;
    A.m0 = 1.0f - t;
}

// The marker's coordinate x (FP64) on a uniform axis: its cell in the box
// [0, size], the axis data of the first RK4 stage and the offsets of the later
// ones (relative to the cell's lower line, in metres).
__device__ __forceinline__ void uni_axis1(double x, double size, double g0, double w, double iw, float fiw, int n,
                                          AxisF &A, AxisRK &R)
{
    const double xc = x < 0 ? 0.0 : (x > size ? size : x);
    const int b = min(max(floor_dm((xc - g0) * iw), 0), n - 2);
    const double gb = fma(dbl_of(b), w, g0);
    uni_tail(n, b, (float)(xc - gb) * fiw, A);
    R.b = b;
    R.du = (float)(x - gb);
    R.lo = (float)(0.0 - gb);
    R.hi = (float)(size - gb);
}

// a later stage point at offset e (metres from the first stage's line)
__device__ __forceinline__ void uni_stage(const AxisRK &R, float e, float fiw, int n, AxisF &A)
{
    if (e < R.lo) e = R.lo;
    if (e > R.hi) e = R.hi;
    const float u = e * fiw;
    int b = R.b + __float2int_rd(u);
    b = min(max(b, 0), n - 2);
    uni_tail(n, b, u - (float)(b - R.b), A);
}

// A later stage point at offset e on a uniform axis (metres from the first
// stage's line, clamped to the box), in half cells: its quarter index along the
// axis (2 b + upper half, within [0, nh - 1]) and its coordinate in that half
// cell.  fiw2 = 2 / width.
__device__ __forceinline__ void uni_half(const AxisRK &R, float e, float fiw2, int nh, int &h, float &f)
{
    e = min_nan(max_nan(e, R.lo), R.hi);
    const float s = e * fiw2;
    float fl;
    const int k0 = 2 * R.b + floor_fm(s, fl);
    const int k = min(max(k0, 0), nh - 1);
    h = k;
    f = s - fl;
    if (k != k0) f = s - (fl - flt_of(k0 - k));  // s - (float)(k - 2 R.b); at the box's edge
}

// vx and vy at a point of quarter cell (hx, hy) with coordinates (fx, fy) in it,
// from the quarter's two forms (GridView.vq4)
__device__ __forceinline__ void quarter_v(const float4 *__restrict__ q, int nhy, int hx, int hy, float fx, float fy,
                                          float &vx, float &vy)
{
    const float4 *p = q + 2 * (hx * nhy + hy);
    const float4 a = __ldg(p), b = __ldg(p + 1);
    const float fxy = fx * fy;
    vx = fmaf(fxy, a.w, fmaf(fy, a.z, fmaf(fx, a.y, a.x)));
    vy = fmaf(fxy, b.w, fmaf(fy, b.z, fmaf(fx, b.y, b.x)));
}

// The mixed RK4 velocity (markmart.c:73-115) on a uniform grid: vx1, vy1 and the
// pressure at the marker, three later stages in FP32 offsets, the stage sum in
// FP64.  X, Y: the first stage's axis data (strain rates of the viscosity update).
__device__ __forceinline__ void rk4_uni(const GridView &G, double x, double y, double dt, int markmod, double &vx0,
                                        double &vy0, double &pr, AxisF &X, AxisF &Y, AxisRK &RX, AxisRK &RY)
{
    const int nx = (int)G.nx, ny = (int)G.ny;
    uni_axis1(x, G.xsize, G.gx0, G.wx, G.iwx, G.fiwx, nx, X, RX);
    uni_axis1(y, G.ysize, G.gy0, G.wy, G.iwy, G.fiwy, ny, Y, RY);
    const double vx1 = (double)bilq(G.vxq, ny, X.b, Y.m, X.b1, Y.m1);
    const double vy1 = (double)bilq(G.vyq, ny, X.m, Y.b, X.m1, Y.b1);
    pr = (double)bilq(G.prq, ny, X.m + 1, Y.m + 1, X.m1, Y.m1);
    if (markmod == 1) {
        vx0 = vx1;
        vy0 = vy1;
        return;
    }
    const float h = (float)(dt / 2.0), f = (float)dt;
    if (G.vq4) {
        // the later stages from the quarter-cell forms: one index and one
        // coordinate per axis instead of the basic and the staggered stencil
        const int nhx = 2 * (nx - 1), nhy = 2 * (ny - 1);
        const float hx2 = 2.0f * G.fiwx, hy2 = 2.0f * G.fiwy;
        int qx, qy;
        float fx, fy, v2x, v2y, v3x, v3y, v4x, v4y;
        uni_half(RX, RX.du + h * (float)vx1, hx2, nhx, qx, fx);
        uni_half(RY, RY.du + h * (float)vy1, hy2, nhy, qy, fy);
        quarter_v(G.vq4, nhy, qx, qy, fx, fy, v2x, v2y);
        uni_half(RX, RX.du + h * v2x, hx2, nhx, qx, fx);
        uni_half(RY, RY.du + h * v2y, hy2, nhy, qy, fy);
        quarter_v(G.vq4, nhy, qx, qy, fx, fy, v3x, v3y);
        uni_half(RX, RX.du + f * v3x, hx2, nhx, qx, fx);
        uni_half(RY, RY.du + f * v3y, hy2, nhy, qy, fy);
        quarter_v(G.vq4, nhy, qx, qy, fx, fy, v4x, v4y);
        constexpr double sixth = 1.0 / 6.0;
        vx0 = (vx1 + 2.0 * (double)v2x + 2.0 * (double)v3x + (double)v4x) * sixth;
        vy0 = (vy1 + 2.0 * (double)v2y + 2.0 * (double)v3y + (double)v4y) * sixth;
        return;
    }
    AxisF Xs, Ys;
    uni_stage(RX, RX.du + h * (float)vx1, G.fiwx, nx, Xs);
    uni_stage(RY, RY.du + h * (float)vy1, G.fiwy, ny, Ys);
    const float v2x = bilq(G.vxq, ny, Xs.b, Ys.m, Xs.b1, Ys.m1), v2y = bilq(G.vyq, ny, Xs.m, Ys.b, Xs.m1, Ys.b1);
    uni_stage(RX, RX.du + h * v2x, G.fiwx, nx, Xs);
    uni_stage(RY, RY.du + h * v2y, G.fiwy, ny, Ys);
    const float v3x = bilq(G.vxq, ny, Xs.b, Ys.m, Xs.b1, Ys.m1), v3y = bilq(G.vyq, ny, Xs.m, Ys.b, Xs.m1, Ys.b1);
    uni_stage(RX, RX.du + f * v3x, G.fiwx, nx, Xs);
    uni_stage(RY, RY.du + f * v3y, G.fiwy, ny, Ys);
    const float v4x = bilq(G.vxq, ny, Xs.b, Ys.m, Xs.b1, Ys.m1), v4y = bilq(G.vyq, ny, Xs.m, Ys.b, Xs.m1, Ys.b1);
    constexpr double sixth = 1.0 / 6.0;
    vx0 = (vx1 + 2.0 * (double)v2x + 2.0 * (double)v3x + (double)v4x) * sixth;
    vy0 = (vy1 + 2.0 * (double)v2y + 2.0 * (double)v3y + (double)v4y) * sixth;
}

// ----------------------------------------------------------------- move + record
__device__ __forceinline__ unsigned lane_lt()
{
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// The 16-byte averaging record {x word, y word, T, log-viscosity word}:
//   x word: w1 of x in [0, 1] as fixed point w1 2^24 (bits 0-24), log-viscosity bits 25-31 (25-31)
//   y word: w1 of y likewise (bits 0-24), log-viscosity bits 21-24 (25-28), immobile
//           (bit 29), type slot (bits 30-31)
//   T: the marker temperature, FP32
//   the last word: log-viscosity bits 32-63
// The log-viscosity is rounded to its 43 leading bits (sign, exponent, 31
// fraction bits: 2.3e-10 of itself); the cell sums turn w1 back into an FP64
// number with one FMA, exactly, and take every field apart with at most three
// bit operations.
constexpr uint32_t kWeightMask = 0x1FFFFFFu;
constexpr uint32_t kRecImmobile = 1u << 29;
constexpr int kRecSlotShift = 30;
// What k_move_fused reads per rock type, a byte: rec_type_byte of an averaged type, and
// bit 0 for a type that movemark leaves where it is (markim)
constexpr int kMoveTypes = 128;
// tinfo[] of a rock type (slot | immobile << 2) as the y word's top byte has it
__host__ __device__ constexpr uint8_t rec_type_byte(uint8_t tinfo)
{
    return (uint8_t)((tinfo & 3u) << 6 | (tinfo & 4u) << 3);
}
__device__ __forceinline__ uint32_t weight_fix(double w)
{
    // w 2^24 + 1.5 x 2^52 rounds to nearest-even at unit resolution, its low word the
    // signed result: __double2int_rn(w 2^24), held to [0, 2^24]
    return (uint32_t)min(max(__double2loint(fma(w, 0x1p24, 0x1.8p52)), 0), 1 << 24);
}
__device__ __forceinline__ double weight_of(uint32_t word)
{
    // (2^52 + n) 2^-24 - 2^28 = n 2^-24, exactly
    return fma(__hiloint2double(0x43300000, (int)(word & kWeightMask)), 0x1p-24, -0x1p28);
}
__device__ __forceinline__ float4 rec_with_lnu(float4 r, double lnu)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(lnu) + (1ull << 20);
    const uint32_t lo = (uint32_t)b, hi = (uint32_t)(b >> 32);
    const uint32_t x = (__float_as_uint(r.x) & kWeightMask) | (lo & ~kWeightMask);
    const uint32_t y = (__float_as_uint(r.y) & ~0x1E000000u) | ((lo << 4) & 0x1E000000u);
    return make_float4(__uint_as_float(x), __uint_as_float(y), r.z, __uint_as_float(hi));
}
// type: the rock type's rec_type_byte
__device__ __forceinline__ float4 rec_pack(uint32_t wx, uint32_t wy, float tk, uint32_t type, double lnu)
{
    return rec_with_lnu(make_float4(__uint_as_float(wx), __uint_as_float(wy | type << 24), tk, 0.f), lnu);
}
__device__ __forceinline__ double rec_lnu(uint32_t x, uint32_t y, uint32_t w)
{
    return __hiloint2double((int)w, (int)((x & ~kWeightMask) | ((y >> 4) & 0x01E00000u)));
}
__device__ __forceinline__ double rec_lnu(float4 r)
{
    return rec_lnu(__float_as_uint(r.x), __float_as_uint(r.y), __float_as_uint(r.w));
}
__device__ __forceinline__ int rec_slot(float4 r) { return (int)(__float_as_uint(r.y) >> kRecSlotShift); }
__device__ __forceinline__ bool rec_immobile(float4 r) { return (__float_as_uint(r.y) & kRecImmobile) != 0; }

// The place of record `slot` of a cell's bucket: buckets of 32 consecutive cells are
// interleaved by pairs of records (a 32-byte sector), so that a warp that reads the
// same pair of 32 neighbouring cells reads 1 KB in a row.  cap is even.
__host__ __device__ __forceinline__ int32_t rec_place(int32_t cell, int32_t slot, int32_t cap)
{
    return (cell >> 5) * (cap << 5) + ((slot >> 1) << 6) + ((cell & 31) << 1) + (slot & 1);
}

// the log-viscosity of a record from the marker's viscosity (the radmax override
// first, markmart.c:335-340), in the form viscmod asks for
__device__ __forceinline__ double record_lnu(const GridView &G, const AvgArgsK &V, double x, double y, double mnu)
{
    if (outside_radmax(G, V, x, y)) mnu = 1.000e+22;
    return V.viscmod == 1 ? log_mixed(mnu) : (V.viscmod == 2 ? 1.0 / mnu : mnu);
}

// per-thread maxima of the call's quantisation bounds: largest cell count, |tk|
// and |log-viscosity| (FP32 bit patterns of upper bounds)
struct FusedStat {
    uint32_t cnt, tk, lnu;
};

// One marker (slot i; live = i < n) of the fused step: movemark from its loaded
// x, y, T, eta and type, then the averaging record at the new cell.  Every lane of
// the warp calls it together (the bucket places are claimed per warp).
template <bool VISC, bool UNI>
__device__ __forceinline__ void move_record(const GridView &G, const MarkerView &M, const i2g_types &T,
                                            const MoveArgs &A, const FusedMove &F, const ViscType *VT,
                                            const uint8_t *type, int64_t i, bool live, int mt, double x, double y,
                                            const double Tm, double eta, FusedStat &st)
{
    const int lane = threadIdx.x & 31;
    bool ok = false, defer = false;
    int32_t key = 0;
    int bx = 0, by = 0;
    float4 rec = make_float4(0.f, 0.f, 0.f, 0.f);
    double lnu = 0.0;
    if (live) {
        // (movemark changes T only for markers that leave the box, which the
        // averaging skips, and eta only with the viscosity update, which reads it
        // again)
        const bool inbox = (x >= 0 && y >= 0 && x <= G.xsize && y <= G.ysize);
        int hx = -1, hy = -1;
        bool moved = false;
        if ((inbox || A.outgrid != 1) && !(type[mt] & 1u)) {
            double pr, vx0, vy0;
            AxisF X1, Y1;
            if (UNI) {
                AxisRK RX, RY;
                rk4_uni(G, x, y, A.timestep, A.markmod, vx0, vy0, pr, X1, Y1, RX, RY);
                hx = RX.b;
                hy = RY.b;
            } else {
                rk4_mixed(G, x, y, A.timestep, A.markmod, vx0, vy0, &pr, hx, hy, VISC ? &X1 : nullptr,
                          VISC ? &Y1 : nullptr);
            }
            M.p[i] = pr;
            if (VISC) {
                double e[6];
                strain_mixed(G, x, y, X1, Y1, e);
                eta = visc_update_mixed(M, T, VT[mt < 20 ? mt : min(mt - 20, kAvgTypes - 1)], A, i, mt, Tm, eta, pr, e);
            }
            if (A.outgrid == 2 && !inbox) {
                if (x < 0 || x > G.xsize) vy0 = 0;
                if (y < 0 || y > G.ysize) vx0 = 0;
            }
            x = advance(x, A.timestep, vx0, A.f32pos);
            y = advance(y, A.timestep, vy0, A.f32pos);
            M.x[i] = x;
            M.y[i] = y;
            moved = true;
        }
        // the averaging's filter at the new position (markmart.c:277)
        const AvgArgsK &V = F.avg;
        const bool inner = x > 0 && y > 0 && x < G.xsize && y < G.ysize;
        if (!inner && moved && (x < 0 || y < 0 || x > G.xsize || y > G.ysize)) M.T[i] = 0;
        ok = inner && Tm > 0 && mt < kAvgTypes && (V.gridmod <= 1 || (M.id[i] % V.gridmod) == 0);
        if (ok) {
            if (UNI) {
                bx = min(max(floor_dm((x - G.gx0) * G.iwx), 0), (int)G.nx - 2);
                by = min(max(floor_dm((y - G.gy0) * G.iwy), 0), (int)G.ny - 2);
            } else {
                bx = hx >= 0 ? cell_walk(G.gx, (int)G.nx, hx, x) : (int)cell_search(G.gx, G.nx, G.inv_x, x);
                by = hy >= 0 ? cell_walk(G.gy, (int)G.ny, hy, y) : (int)cell_search(G.gy, G.ny, G.inv_y, y);
            }
            key = bx * (int32_t)(G.ny - 1) + by;
        }
    }
    // a place in the cell's bucket: warp-aggregated counting atomics, issued
    // before the record is formed so that their round trip overlaps it
    const unsigned okm = __ballot_sync(0xffffffffu, ok);
    unsigned peers = 0;
    int32_t base = 0;
    if (ok) {
        peers = __match_any_sync(okm, key);
        if (lane == __ffs(peers) - 1) base = atomicAdd(F.count + key, __popc(peers));
        // the record: fixed-point weights at the new position, temperature, type
        // slot, log-viscosity
        const AvgArgsK &V = F.avg;
        double wx1, wy1;
        if (UNI) {
            wx1 = (x - fma(dbl_of(bx), G.wx, G.gx0)) * G.iwx;
            wy1 = (y - fma(dbl_of(by), G.wy, G.gy0)) * G.iwy;
        } else {
            wx1 = (x - __ldg(G.gx + bx)) * (double)__ldg(G.ixb + bx);
            wy1 = (y - __ldg(G.gy + by)) * (double)__ldg(G.iyb + by);
        }
        // sticky air held at the ambient temperature (markmart.c:296-309): the
        // record carries it now, the marker's own T is reset by the averaging call
        double mtk = Tm;
        if (mt < 2) {
            mtk = V.tmp_ambient;
            if (Tm != mtk) F.treset[atomicAdd(&F.ctr->ntreset, 1)] = (int32_t)i;
        }
        // a marker without a viscosity of its own (eta <= 0) gets it from
        // viscalc in k_fused_begin (a place is kept for it here)
        lnu = eta > 0 ? record_lnu(G, V, x, y, eta) : 0.0;
        defer = !(eta > 0);
        rec = rec_pack(weight_fix(wx1), weight_fix(wy1), (float)mtk, (uint32_t)(type[mt] & 0xFEu), lnu);
    }
    uint32_t cnt = 0;
    if (ok) {
        base = __shfl_sync(peers, base, __ffs(peers) - 1);
        const int32_t slot = base + __popc(peers & lane_lt());
        cnt = (uint32_t)slot + 1u;
        int32_t place;  // bucket place, or -(overflow index + 1)
        if (slot < F.cap) {
            place = rec_place(key, slot, F.cap);
            F.ra[place] = rec;
        } else {
            const int32_t o = atomicAdd(&F.ctr->novf, 1);
            if (o == 0) *(volatile int32_t *)F.spilled = 1;
            F.ovf[o].a = rec;
            F.ovf[o].cell = key;
            place = -(o + 1);
        }
        if (defer) F.defer[atomicAdd(&F.ctr->ndefer, 1)] = make_int2((int32_t)i, place);
    }
    // the warp's bounds into its running maxima (lane 0)
    if (okm) {
        const uint32_t m0 = __reduce_max_sync(0xffffffffu, cnt);
        const uint32_t m1 = __reduce_max_sync(0xffffffffu, ok ? __float_as_uint(fabsf(rec.z)) : 0u);
        const uint32_t m2 = __reduce_max_sync(0xffffffffu, ok ? __float_as_uint(__double2float_ru(fabs(lnu))) : 0u);
        if (lane == 0) {
            st.cnt = max(st.cnt, m0);
            st.tk = max(st.tk, m1);
            st.lnu = max(st.lnu, m2);
        }
    }
}

// the warp's bounds (lane 0) into one of kFusedParts slots (an atomic only where
// the value exceeds the slot's)
__device__ __forceinline__ void fused_stat_flush(const FusedStat &st, FusedCounters *ctr)
{
    const uint32_t m0 = st.cnt, m1 = st.tk, m2 = st.lnu;
    if ((threadIdx.x & 31) == 0 && m0 > 0) {
        uint32_t *dst = ctr->part[(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) % kFusedParts];
        if (m0 > *(volatile uint32_t *)(dst + 0)) atomicMax(dst + 0, m0);
        if (m1 > *(volatile uint32_t *)(dst + 1)) atomicMax(dst + 1, m1);
        if (m2 > *(volatile uint32_t *)(dst + 2)) atomicMax(dst + 2, m2);
    }
}

// k_move_fused's tiles: 256 markers, one per thread; x, y, T, eta of the next
// tile are copied into shared memory (cp.async, 8 bytes per field and thread)
// while the current one is computed, the type is loaded a tile ahead into a
// register
constexpr int kMoveTile = 256;
struct MoveStage {
    double v[4][kMoveTile];  // x, y, T, eta
};

__device__ __forceinline__ void cp_async8(double *smem, const double *gmem)
{
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem) : "memory");
}

__device__ __forceinline__ void move_stage_issue(const MarkerView &M, MoveStage &S, int64_t i)
{
    if (i < M.n) {
        const int t = threadIdx.x;
        cp_async8(&S.v[0][t], M.x + i);
        cp_async8(&S.v[1][t], M.y + i);
        cp_async8(&S.v[2][t], M.T + i);
        cp_async8(&S.v[3][t], M.eta + i);
    }
    cp_async_commit();
}

// Persistent: CTA b takes tiles b, b + gridDim.x, ... (the grid is the resident
// CTAs of the device, one wave), so the loads of the next tile are in flight
// while the current tile computes.  Each thread copies and reads only its own
// marker's fields: the cp.async group wait orders them, no CTA barrier.  With the
// viscosity update a thread reads the marker its class order gives it, behind the
// order's barriers.  Viscosity update, nonuniform grid, 4M markers: 564 us with
// viscalc's own expressions and searches and walks by the whole axis, 348 with
// viscalc_mixed and the class order (two or three CTAs per SM 401, five 350), 284 with
// the axis bins and branch-free stage steps; viscalc_mixed's powers as pow, for its
// precision, have added 11 since.  Uniform grid without the update, 401^2 nodes, 2.56M
// markers: 69.0 -> 67.0 us and 624 -> 604 instructions per warp and tile with the types'
// flags in shared memory, the box tests shared, and clamps of one instruction.
template <bool VISC, bool UNI>
__global__ void __launch_bounds__(kMoveTile, 4) k_move_fused(const __grid_constant__ GridView G,
                                                    const __grid_constant__ MarkerView M,
                                                    const DevTypes *__restrict__ Ty, const __grid_constant__ MoveArgs A,
                                                    const __grid_constant__ FusedMove F)
{
    __shared__ MoveStage S[2];
    __shared__ FusedStat wst[kMoveTile / 32];
    // the rheology's per-type constants, and the tile's order by the path it takes
    __shared__ ViscType VT[VISC ? kAvgTypes : 1];
    __shared__ uint8_t order[kMoveTile], types[kMoveTile];
    __shared__ int cnt[kMoveTile / 32][4];
    __shared__ uint8_t type[kMoveTypes];
    allow_next();
    wait_previous();
    if (VISC && threadIdx.x < kAvgTypes) VT[threadIdx.x] = visc_type(Ty->t, threadIdx.x);
    if (threadIdx.x < kMoveTypes)
        type[threadIdx.x] = (threadIdx.x < kAvgTypes ? F.type[threadIdx.x] : 0) | (Ty->t.markim[threadIdx.x] ? 1 : 0);
    __syncthreads();
    const i2g_types &T = Ty->t;
    const int tid = threadIdx.x;
    const int ntiles = (int)((M.n + kMoveTile - 1) / kMoveTile);
    FusedStat &st = wst[tid >> 5];
    if ((tid & 31) == 0) st = FusedStat{0u, 0u, 0u};
    int tile = blockIdx.x;
    int64_t i = (int64_t)tile * kMoveTile + tid;
    move_stage_issue(M, S[0], i);
    int mt_next = i < M.n ? M.type[i] : 0;
    for (int b = 0; tile < ntiles; tile += gridDim.x, b ^= 1) {
        i = (int64_t)tile * kMoveTile + tid;
        const int64_t inext = i + (int64_t)gridDim.x * kMoveTile;
        move_stage_issue(M, S[b ^ 1], inext);
        int mt = mt_next, mine = tid;
        mt_next = inext < M.n ? M.type[inext] : 0;
        cp_async_wait<1>();  // this tile's copies
        if (VISC) {
            // a thread takes a marker of the tile by its rheology's path
            types[tid] = (uint8_t)mt;
            mine = class_order(i < M.n && mt < kAvgTypes ? VT[mt < 20 ? mt : mt - 20].cls : 0, order, cnt);
            mt = (int8_t)types[mine];
            i = (int64_t)tile * kMoveTile + mine;
        }
        const bool live = i < M.n;
        double x = 0.0, y = 0.0, Tm = 0.0, eta = 0.0;
        if (live) {
            x = S[b].v[0][mine];
            y = S[b].v[1][mine];
            Tm = S[b].v[2][mine];
            eta = S[b].v[3][mine];
        }
        move_record<VISC, UNI>(G, M, T, A, F, VT, type, i, live, mt, x, y, Tm, eta, st);
        if (VISC) __syncthreads();  // the tile's stage and order are done with
    }
    cp_async_wait<0>();
    fused_stat_flush(st, F.ctr);
}

// ----------------------------------------------------------------- sums and nodes
// The rounding of one averaging call, derived from the counters: two ways to add
// terms in FP64 so that the sum does not depend on their order.
//   quant   a term t becomes fma(a, b, c) - c, t rounded to the nearest multiple of
//           the quantum q = 2^(e - 52), c = 1.5 * 2^e, where 2^e exceeds the largest
//           magnitude any node's sum can reach (4 x the largest cell count x the
//           largest |term|): every partial sum is an integer multiple of q below
//           2^52 q, an exact FP64 number.  Opposite terms stay opposite.
//   binade  the sum starts at c / 2 and takes each term as fma(a, b, sum): it stays in
//           its binade (a cell's sum is at most a quarter of a node's), where doubles
//           are q / 2 apart, so every term adds its nearest multiple of q / 2, whatever
//           came before it.  Only a tie would depend on that, and there is none: the
//           last fraction bit of one factor is set (odd), so a term is an odd multiple
//           of 2^-52 of that factor's leading bit times the other's last bit; were that
//           2^(e - 54), half the spacing, the term would be 2^(e - 2) or more, where it
//           is below 2^(e - 4).  One FP64 operation per term, half of quant's error.
struct QConst {
    double cw, ctk, cnu;  // weights, temperature x weight, log-viscosity x weight
    // a node goes to node_guard where a weight sum is below thr_w (thr_nuw for
    // the viscosity weights), or |TK| below vtk, or |NU|, |ND| below vnu: there
    // the quanta could move its value by more than 1e-9 of the value
    double thr_w, thr_nuw, vtk, vnu;
};

__device__ __forceinline__ QConst qconst_of(uint32_t cmax, uint32_t tkb, uint32_t lnb, int viscmod)
{
    QConst Q;
    // weights are in [-1, 1]; up to Nn terms reach a node (at least 4 a cell: the
    // cell sums run whole batches)
    const double Nn = 4.0 * (double)(cmax > 4u ? cmax : 4u), Sw = Nn * (1.0 + 0x1p-20);
    const double Mtk = (double)__uint_as_float(tkb), Mnu = (double)__uint_as_float(lnb);
    const double Stk = Sw * Mtk, Snu = Sw * Mnu;
    const int ew = ilogb(Sw) + 1, etk = Stk > 0 ? ilogb(Stk) + 1 : 0, enu = Snu > 0 ? ilogb(Snu) + 1 : 0;
    Q.cw = ldexp(1.5, ew);
    Q.ctk = ldexp(1.5, etk);
    Q.cnu = ldexp(1.5, enu);
    // A node sum of up to Nn terms moves by at most Nn q / 2 (in its binade half of that).  A weighted mean
    // S / W then moves by at most (Nn q_S / 2) / |S| + (Nn q_w / 2) / W of
    // itself; keep each part below 1e-9.  For log-viscosity (viscmod 1) the mean
    // is an exponent: its absolute error, (Nn q_S / 2 + |mean| Nn q_w / 2) / W,
    // is the relative error of the node value.
    const double qw = ldexp(1.0, ew - 52), qtk = ldexp(1.0, etk - 52), qnu = ldexp(1.0, enu - 52);
    Q.thr_w = Nn * qw / 2e-9;
    Q.vtk = 4.0 * Nn * qtk / 2e-9;
    if (viscmod == 1) {
        Q.thr_nuw = Nn * (qnu + qw * Mnu) / 2e-9;
        Q.vnu = 0.0;
    } else {
        Q.thr_nuw = Q.thr_w;
        Q.vnu = Nn * qnu / 2e-9;
    }
    return Q;
}

// the counters' maxima over the kFusedParts slots; every thread of the block
// gets the same QConst (threads 0..63 read, the block reduces in shared memory)
__device__ __forceinline__ QConst block_qconst(const FusedCounters *ctr, int viscmod)
{
    __shared__ uint32_t s[3][2];
    __shared__ QConst sq;
    const int t = threadIdx.x;
    uint32_t a = 0, b = 0, c = 0;
    if (t < kFusedParts) {
        a = ctr->part[t][0];
        b = ctr->part[t][1];
        c = ctr->part[t][2];
    }
    if (t < 64) {
        a = __reduce_max_sync(0xffffffffu, a);
        b = __reduce_max_sync(0xffffffffu, b);
        c = __reduce_max_sync(0xffffffffu, c);
        if ((t & 31) == 0) {
            s[0][t >> 5] = a;
            s[1][t >> 5] = b;
            s[2][t >> 5] = c;
        }
    }
    __syncthreads();
    if (t == 0) sq = qconst_of(max(s[0][0], s[0][1]), max(s[1][0], s[1][1]), max(s[2][0], s[2][1]), viscmod);
    __syncthreads();
    return sq;
}

// The sums of one cell.  With x = 2 X1 - 1, y = 2 Y1 - 1 in [-1, 1] a record's
// corner weights are (1 -+ x)(1 -+ y) / 4, so a cell needs, per type slot, the record
// count and the sums of x, y and x y, and for the mobile records T, T x, T y and
// T x y; corner4 turns them into the sums at a corner.  The node viscosity goes to
// the nearest node with the quadrant weight |x y|, the cell-centre one with the tent
// weight (1 - |x|)(1 - |y|).
//
// No sum is picked per record (a predicated FP64 add became two selects): sums over a
// part of the records come from sums with signs.  With s1, s2 = -1 where bit 0, 1 of
// the slot is set, else 1, the sums of f, s1 f and s2 f (and s1 s2 f with four slots)
// give every slot's, and those of t, sx t, sy t and sx sy t (sx, sy the signs of x, y)
// every quadrant's, exactly, for quantized f and t.
template <int NT>
struct CellAcc {
    static constexpr int B = NT == 1 ? 0 : (NT == 2 ? 1 : (NT == 3 ? 2 : 3));  // signed copies of the slot sums
    int32_t m[B + 1];                      // records with bit 0, bit 1, both bits set (B of them)
    double x[B + 1], y[B + 1], p[B + 1];   // x, y, x y (quantized): plain, s1, s2, s1 s2
    double w, wx, wy;                      // |x y| plain, sx, sy (sx sy: p[0])
    double n[4];                           // log-viscosity x |x y| (quantized): plain, sx, sy, sx sy
    double t0, tx, ty, txy, nd, wnd;       // sums in their binade
};

template <int NT>
__device__ __forceinline__ void acc_start(CellAcc<NT> &a, const QConst &Q)
{
#pragma unroll
    for (int k = 0; k <= CellAcc<NT>::B; k++) {
        a.m[k] = 0;
        a.x[k] = a.y[k] = a.p[k] = 0.0;
    }
    a.w = a.wx = a.wy = 0.0;
#pragma unroll
    for (int k = 0; k < 4; k++) a.n[k] = 0.0;
    a.t0 = a.tx = a.ty = a.txy = 0.5 * Q.ctk;
    a.nd = 0.5 * Q.cnu;
    a.wnd = 0.5 * Q.cw;
}

// +-1.0 with the sign bit of word b
__device__ __forceinline__ double unit_of(uint32_t b)
{
    return __hiloint2double((int)((b & 0x80000000u) | 0x3FF00000u), 0);
}

// v with its last fraction bit set, one unit more for the terms below (their last bits
// are zero: 24-bit numbers and products of two); 0 becomes the smallest subnormal, which
// adds nothing to a sum
__device__ __forceinline__ double odd(double v)
{
    return __hiloint2double(__double2hiint(v), __double2loint(v) | 1);
}

// One record into its cell's sums (markmart.c:859-913): 32 FP64 operations with three
// slots.
template <int NT>
__device__ __forceinline__ void acc_rec(CellAcc<NT> &a, uint4 u, const QConst &Q)
{
    constexpr int B = CellAcc<NT>::B;
    // (2^52 + X) 2^-23 - 2^29 - 1 = 2 X1 - 1, exactly
    const double x = fma(__hiloint2double(0x43300000, (int)(u.x & kWeightMask)), 0x1p-23, -(0x1p29 + 1.0));
    const double y = fma(__hiloint2double(0x43300000, (int)(u.y & kWeightMask)), 0x1p-23, -(0x1p29 + 1.0));
    const double xy = x * y;  // 24 x 24 bits: exact
    const double p = (xy + Q.cw) - Q.cw;
    a.x[0] += x;
    a.y[0] += y;
    a.p[0] += p;
#pragma unroll
    for (int k = 1; k <= B; k++) {
        const uint32_t bit = k == 1 ? u.y << 1 : (k == 2 ? u.y : u.y & (u.y << 1));
        a.m[k - 1] += (int32_t)(bit >> 31);
        const double s = unit_of(k < 3 ? bit : u.y ^ (u.y << 1));
        a.x[k] = fma(s, x, a.x[k]);
        a.y[k] = fma(s, y, a.y[k]);
        a.p[k] = fma(s, p, a.p[k]);
    }
    // the temperature of mobile types
    const double tk = odd((double)__uint_as_float(u.y & kRecImmobile ? 0u : u.z));
    a.t0 += tk;
    a.tx = fma(tk, x, a.tx);
    a.ty = fma(tk, y, a.ty);
    a.txy = fma(tk, xy, a.txy);
    // the nearest node takes the viscosity with the quadrant weight
    // 4 (wa - 1/2)(wb - 1/2), wa = max(X0, X1) = (1 + |x|) / 2 (zero on a midline)
    const double lnu = rec_lnu(u.x, u.y, u.w);
    const uint32_t bx = (uint32_t)__double2hiint(x), by = (uint32_t)__double2hiint(y);
    const double sx = unit_of(bx), sy = unit_of(by);
    a.w += fabs(p);
    a.wx = fma(p, sy, a.wx);  // |x y| sx = x y sy
    a.wy = fma(p, sx, a.wy);
    const double t = fma(lnu, fabs(xy), Q.cnu) - Q.cnu;
    a.n[0] += t;
    a.n[1] = fma(t, sx, a.n[1]);
    a.n[2] = fma(t, sy, a.n[2]);
    a.n[3] = fma(t, unit_of(bx ^ by), a.n[3]);
    // the cell centre takes it with the tent weight 4 (dx - 1/2)(dy - 1/2),
    // dx = 1 - |X0 - 1/2| = 1 - |x| / 2
    const double c = odd((1.0 - fabs(x)) * (1.0 - fabs(y)));
    a.nd = fma(lnu, c, a.nd);
    a.wnd += c;
}

// a record whose terms are zero in every sum but wnd (there 1, 2^-52 being less than
// half of any q / 2): x = y = T = 0, lnu = 0
__device__ __forceinline__ uint4 rec_none() { return make_uint4(1u << 23, 1u << 23, 0u, 0u); }

struct RecPair {
    uint4 a, b;
};
__device__ __forceinline__ RecPair rec_pair(const uint4 *p)
{
    RecPair r;
    r.a = __ldcs(p);
    r.b = __ldcs(p + 1);
    return r;
}
// the pair of records at p of which m (<= 0: none) are there
__device__ __forceinline__ RecPair rec_pair(const uint4 *p, int m)
{
    RecPair r;
    r.a = r.b = rec_none();
    if (m > 0) r.a = __ldcs(p);
    if (m > 1) r.b = __ldcs(p + 1);
    return r;
}

// A cell's sums as k_cellnodes keeps them in shared memory: per slot {n, x, y, xy},
// then {T, T x, T y, T x y}, nu[4], wnu[4], nd, wnd.
template <int NT>
struct CellSums {
    static constexpr int T = 4 * NT, NU = T + 4, WNU = NU + 4, ND = WNU + 4, WND = ND + 1, N = WND + 1;
};

// the sums of S neighbouring lanes, each lane of them the total
template <int S, class V>
__device__ __forceinline__ V lanes_sum(V v)
{
#pragma unroll
    for (int o = 1; o < S; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// out(f, value) for every field f of CellSums from a cell's sums over S lanes; n: the
// cell's records
template <int NT, int S, class Out>
__device__ __forceinline__ void acc_finish(CellAcc<NT> &a, const QConst &Q, int32_t n, Out &&out)
{
    using C = CellSums<NT>;
    constexpr int B = CellAcc<NT>::B;
    int32_t m[3] = {0, 0, 0};
#pragma unroll
    for (int k = 0; k < B; k++) m[k] = lanes_sum<S>(a.m[k]);
#pragma unroll
    for (int f = 0; f < 4; f++) {
        double v[4] = {0.0, 0.0, 0.0, 0.0};  // the sum and its signed copies
        if (f == 0) {
            v[0] = (double)n;
#pragma unroll
            for (int k = 1; k <= B; k++) v[k] = k < 3 ? (double)(n - 2 * m[k - 1]) : (double)(n - 2 * (m[0] + m[1] - 2 * m[2]));
        } else {
#pragma unroll
            for (int k = 0; k <= B; k++) v[k] = lanes_sum<S>(f == 1 ? a.x[k] : (f == 2 ? a.y[k] : a.p[k]));
        }
        if (NT == 1) out(f, v[0]);
        if (NT == 2) {
            out(f, 0.5 * (v[0] + v[1]));
            out(4 + f, 0.5 * (v[0] - v[1]));
        }
        if (NT == 3) {  // slots 0, 1, 2: (s1, s2) = (+, +), (-, +), (+, -)
            out(f, 0.5 * (v[1] + v[2]));
            out(4 + f, 0.5 * (v[0] - v[1]));
            out(8 + f, 0.5 * (v[0] - v[2]));
        }
        if (NT == 4) {
            out(f, 0.25 * ((v[0] + v[1]) + (v[2] + v[3])));
            out(4 + f, 0.25 * ((v[0] - v[1]) + (v[2] - v[3])));
            out(8 + f, 0.25 * ((v[0] + v[1]) - (v[2] + v[3])));
            out(12 + f, 0.25 * ((v[0] - v[1]) - (v[2] - v[3])));
        }
        if (f == 3) a.p[0] = v[0];
    }
    out(C::T, lanes_sum<S>(a.t0 - 0.5 * Q.ctk));
    out(C::T + 1, lanes_sum<S>(a.tx - 0.5 * Q.ctk));
    out(C::T + 2, lanes_sum<S>(a.ty - 0.5 * Q.ctk));
    out(C::T + 3, lanes_sum<S>(a.txy - 0.5 * Q.ctk));
    const double n0 = lanes_sum<S>(a.n[0]), n1 = lanes_sum<S>(a.n[1]), n2 = lanes_sum<S>(a.n[2]),
                 n3 = lanes_sum<S>(a.n[3]);
    out(C::NU + 0, 0.25 * ((n0 - n1) - (n2 - n3)));
    out(C::NU + 1, 0.25 * ((n0 - n1) + (n2 - n3)));
    out(C::NU + 2, 0.25 * ((n0 + n1) - (n2 + n3)));
    out(C::NU + 3, 0.25 * ((n0 + n1) + (n2 + n3)));
    const double w0 = lanes_sum<S>(a.w), w1 = lanes_sum<S>(a.wx), w2 = lanes_sum<S>(a.wy), w3 = a.p[0];
    out(C::WNU + 0, 0.25 * ((w0 - w1) - (w2 - w3)));
    out(C::WNU + 1, 0.25 * ((w0 - w1) + (w2 - w3)));
    out(C::WNU + 2, 0.25 * ((w0 + w1) - (w2 + w3)));
    out(C::WNU + 3, 0.25 * ((w0 + w1) + (w2 + w3)));
    out(C::ND, lanes_sum<S>(a.nd - 0.5 * Q.cnu));
    out(C::WND, lanes_sum<S>(a.wnd - 0.5 * Q.cw));
}

// 4 x the sum at corner q = 2a + b (node (m1 + a, m2 + b)) of a bilinear quadruple
// {1, x, y, xy} sum; c: distance between the four in memory
template <int q>
__device__ __forceinline__ double corner4(const double *v, int c)
{
    const double s = v[0], x = v[c], y = v[2 * c], xy = v[3 * c];
    if (q == 0) return ((s - x) - y) + xy;
    if (q == 1) return ((s - x) + y) - xy;
    if (q == 2) return ((s + x) - y) - xy;
    return ((s + x) + y) + xy;
}

struct CellNodesArgs {
    int32_t nx, ny, nc1, nc2, cap;
    uint32_t mob;  // bit k set when type slot k's type is mobile (its T is averaged)
    int32_t ncol;  // node columns per CTA: kCnCols * groups - 1
    int32_t ntx;   // CTAs along x
    const int32_t *count;
    const float4 *ra;
    const OvfRec *ovf;
    FusedCounters *ctr;
    double sv[4][4];  // per type slot: ro, cp, kt, ht
    int32_t plain;    // none of them is above 2^500 or no number (div_by's means)
    // a step replayed from a CUDA graph: the slots' radiogenic heat from the
    // step's row of a device table (stepc[4 * *stepi + group] x density, group
    // 1..3 = silicate, iron, chondrite, 0 = none) instead of sv[.][3]; NULL otherwise
    const double *stepc;
    const int32_t *stepi;
    double sro[4];
    int32_t sgrp[4];
    int32_t viscmod;
    double nubeg, nuend;
    const double *mu;
    NodeOut O;
    unsigned long long *navg;  // averaged markers (the records of the cells a CTA owns)
};

// The sums a node is made of: per-slot weights wt[NT], w1, tk, nu, wnu, nd, wnd
template <int NT>
struct NodeVals {
    static constexpr int N = NT + 6;
};

__device__ __forceinline__ unsigned long long okey(double v)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}
__device__ __forceinline__ double okey_inv(unsigned long long k)
{
    return __longlong_as_double((long long)((k >> 63) ? (k & 0x7fffffffffffffffull) : ~k));
}

__device__ __forceinline__ double visc_finish(int viscmod, double v)
{
    if (viscmod == 1) v = exp(v);
    if (viscmod == 2) v = 1.0 / v;
    return v;
}

// Node m3 from its sums (markmart.c:917-993), the FP64 node loop: viscosity at
// the node (quadrant sums) and at the cell centre (nd), then the weighted means.
// S: per-slot weights wt[NT], w1, tk, nu, wnu, nd, wnd.
// The type slots' radiogenic heat of this call (sv[.][3]) or, for a step replayed
// from a graph, of the step's row of the device table, in shared memory: the
// block's first threads write it, the block syncs before node_write reads it.
__device__ __forceinline__ double *slot_heat()
{
    __shared__ double h[kFusedSlots];
    return h;
}
__device__ __forceinline__ void slot_heat_init(const CellNodesArgs &P)
{
    if (threadIdx.x < kFusedSlots) {
        const int s = threadIdx.x;
        double v = P.sv[s][3];
        if (P.stepc) {
            const int g = P.sgrp[s];
            const double rad = g ? P.stepc[4 * *P.stepi + g] : 0.0;
            v = rad * P.sro[s];  // rad_of(type) x density, as the host forms sv[.][3]
        }
        slot_heat()[s] = v;
    }
}

template <int NT>
__device__ __forceinline__ void node_write(const CellNodesArgs &P, int64_t m3, const double *S, double &vmin,
                                           double &vmax, int &any)
{
    double W0 = 0.0;
#pragma unroll
    for (int k = 0; k < NT; k++) W0 += S[k];
    const double W1 = S[NT], TK = S[NT + 1], NU = S[NT + 2], WNU = S[NT + 3], ND = S[NT + 4], WND = S[NT + 5];
    const double mu = P.mu ? __ldg(P.mu + m3) : 0.0;
    if (WNU != 0.0) {
        double v = mu ? mu : visc_finish(P.viscmod, NU / WNU);
        if (v < P.nubeg) v = P.nubeg;
        if (v > P.nuend) v = P.nuend;
        if (!any) { vmin = vmax = v; any = 1; }
        else { vmin = fmin(vmin, v); vmax = fmax(vmax, v); }
        P.O.nu[m3] = v;
    }
    if (WND != 0.0) {
        double v = mu ? mu : visc_finish(P.viscmod, ND / WND);
        if (v < P.nubeg) v = P.nubeg;
        if (v > P.nuend) v = P.nuend;
        if (!any) { vmin = vmax = v; any = 1; }
        else { vmin = fmin(vmin, v); vmax = fmax(vmax, v); }
        P.O.nd[m3] = v;
        P.O.po[m3] = 0.0;  // po0[] is never accumulated (markmart.c:968)
    }
    if (W0 != 0.0) {
        double r = 0.0, c = 0.0, k = 0.0, h = 0.0;
#pragma unroll
        for (int s = 0; s < NT; s++) {
            r += P.sv[s][0] * S[s];
            c += P.sv[s][1] * S[s];
            k += P.sv[s][2] * S[s];
            h += slot_heat()[s] * S[s];
        }
        // the quotients over one reciprocal (a weight sum is at least one quantum: within
        // div_by's range)
        const double iw = 1.0 / W0;
        auto mean = [&](double v) { return P.plain ? div_by(v, W0, iw) : v / W0; };
        P.O.ro[m3] = mean(r);
        P.O.et[m3] = 0.0;  // beta is zero on constant-property calls
        P.O.cp[m3] = mean(c);
        P.O.kt[m3] = mean(k);
        P.O.ht[m3] = mean(h);
        if (W1 != 0.0) P.O.tk[m3] = TK / W1;
    }
}

// A node whose sums are so small that the call's quanta would cost more than
// 1e-9 of a value is left to node_guard (true).
template <int NT>
__device__ __forceinline__ bool node_finish(const CellNodesArgs &P, const QConst &Q, int m1, int m2, const double *S,
                                            double &vmin, double &vmax, int &any)
{
    const int64_t m3 = (int64_t)m1 * P.ny + m2;
    double W0 = 0.0;
#pragma unroll
    for (int k = 0; k < NT; k++) W0 += S[k];
    const double W1 = S[NT], TK = S[NT + 1], NU = S[NT + 2], WNU = S[NT + 3], ND = S[NT + 4], WND = S[NT + 5];
    const bool flag = (W0 > 0 && W0 < Q.thr_w) || (W1 > 0 && (W1 < Q.thr_w || fabs(TK) < Q.vtk)) ||
                      (WNU > 0 && (WNU < Q.thr_nuw || fabs(NU) < Q.vnu)) ||
                      (WND > 0 && (WND < Q.thr_nuw || fabs(ND) < Q.vnu));
    if (!flag) node_write<NT>(P, m3, S, vmin, vmax, any);
    return flag;
}

// {min, max, any} of the CTA into the call's ordered-key atomics
__device__ __forceinline__ void fold_minmax(double vmin, double vmax, int any, FusedCounters *ctr,
                                            unsigned cnt = 0, unsigned long long *navg = nullptr)
{
    __shared__ double smin[32], smax[32];
    __shared__ int sany[32];
    if (navg) {
        for (int o = 16; o > 0; o >>= 1) cnt += __shfl_down_sync(0xffffffffu, cnt, o);
        if ((threadIdx.x & 31) == 0 && cnt) atomicAdd(navg, (unsigned long long)cnt);
    }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int o = 16; o > 0; o >>= 1) {
        const double a2 = __shfl_down_sync(0xffffffffu, vmin, o), b2 = __shfl_down_sync(0xffffffffu, vmax, o);
        const int c2 = __shfl_down_sync(0xffffffffu, any, o);
        if (c2) {
            if (!any) { vmin = a2; vmax = b2; any = 1; }
            else { vmin = fmin(vmin, a2); vmax = fmax(vmax, b2); }
        }
    }
    __syncthreads();
    if (lane == 0) { smin[w] = vmin; smax[w] = vmax; sany[w] = any; }
    __syncthreads();
    if (threadIdx.x == 0) {
        double a = 0, b = 0;
        int c = 0;
        for (int i = 0; i < (int)(blockDim.x >> 5); i++) {
            if (!sany[i]) continue;
            if (!c) { a = smin[i]; b = smax[i]; c = 1; }
            else { a = fmin(a, smin[i]); b = fmax(b, smax[i]); }
        }
        if (c) {
            atomicMin(&ctr->kmin, okey(a));
            atomicMax(&ctr->kmax, okey(b));
            if (!ctr->any) atomicExch(&ctr->any, 1);
        }
    }
}

// The viscosity range of the nodes a thread wrote
struct ViscRange {
    double lo, hi;
    int any;
};

// A node whose sums are small against the call's quanta, by a warp: the records of
// the node's four cells once for the largest terms, once more with quanta fitted to
// this node (so the sums are exact again, at a resolution of 2^-52 of the node's own
// largest terms), then the node as node_write makes it.
template <int NT>
static __device__ __noinline__ void node_guard(const CellNodesArgs &P, int m1, int m2, ViscRange *range)
{
    const int lane = threadIdx.x & 31;
    const int64_t m3 = (int64_t)m1 * P.ny + m2;
    const int novf = P.ctr->novf;
    constexpr int NV = NT + 6;
    // the terms of a record of cell c (c = 0..3: cells (m1-1, m2-1), (m1-1, m2),
    // (m1, m2-1), (m1, m2)), which reaches the node through its corner 3 - c:
    // t[0] weight, t[1] T x weight, t[2] quadrant weight, t[3] its
    // log-viscosity term, t[4] centre weight, t[5] its term
    auto terms = [&](int c, float4 r, double lnu, double *t) {
        const int q = 3 - c;
        const double X1 = weight_of(__float_as_uint(r.x)), Y1 = weight_of(__float_as_uint(r.y));
        const double X0 = 1.0 - X1, Y0 = 1.0 - Y1;
        const double wx = (q >> 1) ? X1 : X0, wy = (q & 1) ? Y1 : Y0;
        t[0] = wx * wy;
        t[1] = (double)r.z * t[0];
        t[2] = t[3] = t[4] = t[5] = 0.0;
        if (wx > 0.5 && wy > 0.5) {
            t[2] = 4.0 * (wx - 0.5) * (wy - 0.5);
            t[3] = lnu * t[2];
        }
        if (c == 0) {
            const double dx = 1.0 - fabs(X0 - 0.5), dy = 1.0 - fabs(Y0 - 0.5);
            if (dx > 0.5 && dy > 0.5) {
                t[4] = 4.0 * (dx - 0.5) * (dy - 0.5);
                t[5] = lnu * t[4];
            }
        }
    };
    auto each = [&](auto &&fn) {
        for (int c = 0; c < 4; c++) {
            const int c1 = m1 - 1 + (c >> 1), c2 = m2 - 1 + (c & 1);
            if (c1 < 0 || c2 < 0 || c1 >= P.nc1 || c2 >= P.nc2) continue;
            const int64_t cell = (int64_t)c1 * P.nc2 + c2;
            const int32_t n = P.count[cell], nb = min(n, P.cap);
            for (int t = lane; t < nb; t += 32) {
                const float4 r = P.ra[rec_place((int32_t)cell, t, P.cap)];
                fn(c, r, rec_lnu(r));
            }
            if (n > nb)
                for (int o = lane; o < novf; o += 32)
                    if (P.ovf[o].cell == (int32_t)cell) fn(c, P.ovf[o].a, rec_lnu(P.ovf[o].a));
        }
    };
    double mx[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    int nrec = 0;
    each([&](int c, float4 r, double lnu) {
        double t[6];
        terms(c, r, lnu, t);
        for (int k = 0; k < 6; k++) mx[k] = fmax(mx[k], fabs(t[k]));
        nrec++;
    });
    for (int o = 16; o > 0; o >>= 1) {
        for (int k = 0; k < 6; k++) mx[k] = fmax(mx[k], __shfl_xor_sync(0xffffffffu, mx[k], o));
        nrec += __shfl_xor_sync(0xffffffffu, nrec, o);
    }
    double cq[6];
    for (int k = 0; k < 6; k++) {
        const double b = (double)(nrec > 0 ? nrec : 1) * mx[k];
        cq[k] = ldexp(1.5, b > 0 ? ilogb(b) + 1 : 0);
    }
    double S[NV];
    for (int k = 0; k < NV; k++) S[k] = 0.0;
    each([&](int c, float4 r, double lnu) {
        double t[6];
        terms(c, r, lnu, t);
        const double wq = (t[0] + cq[0]) - cq[0];
        const int slot = rec_slot(r);
        for (int k = 0; k < NT; k++)
            if (slot == k) S[k] += wq;
        if (!rec_immobile(r)) {
            S[NT] += wq;
            S[NT + 1] += (t[1] + cq[1]) - cq[1];
        }
        S[NT + 2] += (t[3] + cq[3]) - cq[3];
        S[NT + 3] += (t[2] + cq[2]) - cq[2];
        S[NT + 4] += (t[5] + cq[5]) - cq[5];
        S[NT + 5] += (t[4] + cq[4]) - cq[4];
    });
    for (int o = 16; o > 0; o >>= 1)
        for (int k = 0; k < NV; k++) S[k] += __shfl_xor_sync(0xffffffffu, S[k], o);
    if (lane == 0) node_write<NT>(P, m3, S, range->lo, range->hi, range->any);
}

// One CTA: node rows [d0, d0 + ROWS - 1) x node columns [cs, cs + ncol).  In group g
// warp w takes cell column cs - 1 + 8 g + w: its lanes S to a cell (lane s the pairs
// of records s, s + S, ...), whose sums meet by shuffles and go to shared memory
// (column w + 1; column 0 holds the last one of the group before); then a thread
// finishes a node from its four cells.
//
// Per record and lane 32 FP64 operations and about 75 instructions in all, no branch; a
// cell and its node add about 500 once.  No one resource bounds it: at 13M records and
// 601^2 nodes 53% of the issue slots, 42% of the FP64 pipe and 30% of the DRAM rate
// (18.4 B a record) are in use, with 260 CTAs for 296 places and 16 warps on a full SM;
// a warp runs as long as its fullest cell in whole batches (14% more than the mean after
// five steps at 36 a cell), and waits for its records' loads and its sums' dependent
// steps with few others to fill in.  A lane to a cell reads whole kilobytes (rec_place) and needs no staging; S = 2
// halves the serial chain where a grid leaves the device idle.  Per launch, with the
// kernel that staged the records and picked slots and quadrants by one-hot factors
// (226 instructions per record) before: 36M records, 1001^2 nodes 314 -> 207 us (DRAM
// alone: 120); 2.56M, 401^2 41 -> 30; 160k, 101^2 24.5 -> 8.3; 6400, 21^2 21.7 -> 8.0.
// The means as quotients have added 1 to 2% since.
constexpr int kCnCols = 8, kCnThreads = 32 * kCnCols;
constexpr int kCnBatch = 2;  // pairs of records per batch
template <int NT, int S>
struct CnShape {
    static constexpr int ROWS = 32 / S;
    using C = CellSums<NT>;
    double v[C::N][kCnCols + 1][ROWS];
};
template <int NT, int S>
__global__ void __launch_bounds__(kCnThreads, 2) k_cellnodes(const __grid_constant__ CellNodesArgs P)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    using Shape = CnShape<NT, S>;
    using C = CellSums<NT>;
    Shape &M = *reinterpret_cast<Shape *>(smraw);
    constexpr int ROWS = Shape::ROWS, CS = (kCnCols + 1) * ROWS;
    allow_next();
    wait_previous();
    slot_heat_init(P);  // block_qconst syncs the block
    const QConst Q = block_qconst(P.ctr, P.viscmod);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = lane % S;
    const int cs = (int)(blockIdx.x % P.ntx) * P.ncol, d0 = (int)(blockIdx.x / P.ntx) * (ROWS - 1);
    const int groups = (P.ncol + 1) / kCnCols;
    const uint4 *recs = reinterpret_cast<const uint4 *>(after_wait(P.ra));
    double vmin = 0.0, vmax = 0.0;
    int any = 0;
    unsigned owned = 0;
    const int32_t *count = after_wait(P.count);
    for (int g = 0; g < groups; g++) {
        const int cc = cs - 1 + kCnCols * g + warp;
        const int row = lane / S, cr = d0 - 1 + row;
        const bool valid = cc >= 0 && cc < P.nc1 && cr >= 0 && cr < P.nc2;
        const int64_t cell = (int64_t)cc * P.nc2 + cr;
        const int32_t n = valid ? count[cell] : 0;
        if (sub == 0 && row >= 1 && !(g == 0 && warp == 0)) owned += (unsigned)n;  // each cell counted by one CTA
        const int32_t nb = min(n, P.cap);
        // the lane's pairs of records: sub, sub + S, ...; every lane runs the warp's
        // longest count in whole batches, with records that add nothing but 1 to
        // wnd past its own
        const uint4 *p = recs + (valid ? rec_place((int32_t)cell, 2 * sub, P.cap) : 0);
        const int left = nb - 2 * sub, most = (int)__reduce_max_sync(0xffffffffu, (unsigned)max(left, 0)),
                  whole = (most + 2 * S * kCnBatch - 1) / (2 * S * kCnBatch),
                  least = (int)__reduce_min_sync(0xffffffffu, (unsigned)max(left, 0));
        CellAcc<NT> a;
        acc_start(a, Q);
        RecPair r[kCnBatch];
#pragma unroll
        for (int k = 0; k < kCnBatch; k++) r[k] = rec_pair(p + k * S * 64, left - k * 2 * S);
        for (int i = 1; i <= whole; i++) {
            RecPair u[kCnBatch];
            p += kCnBatch * S * 64;
#pragma unroll
            for (int k = 0; k < kCnBatch; k++) u[k] = r[k];
            if ((i + 1) * kCnBatch * 2 * S <= least) {
#pragma unroll
                for (int k = 0; k < kCnBatch; k++) r[k] = rec_pair(p + k * S * 64);
            } else {
#pragma unroll
                for (int k = 0; k < kCnBatch; k++)
                    r[k] = rec_pair(p + k * S * 64, left - (i * kCnBatch + k) * 2 * S);
            }
#pragma unroll
            for (int k = 0; k < kCnBatch; k++) {
                acc_rec<NT>(a, u[k].a, Q);
                acc_rec<NT>(a, u[k].b, Q);
            }
        }
        // (a lane's own records: its whole pairs, and the odd last one)
        const int own = left <= 0 ? 0 : (left / (2 * S)) * 2 + min(left % (2 * S), 2);
        a.wnd -= (double)(whole * kCnBatch * 2 - own);
        if (n > nb) {  // a full bucket: the rest of the cell's records are in the overflow list
            const int novf = P.ctr->novf;
            for (int o = sub; o < novf; o += S)
                if (P.ovf[o].cell == (int32_t)cell) acc_rec<NT>(a, *reinterpret_cast<const uint4 *>(&P.ovf[o].a), Q);
        }
        __syncwarp();
        acc_finish<NT, S>(a, Q, n, [&](int f, double v) {
            if (f % S == sub) M.v[f][warp + 1][row] = v;
        });
        __syncthreads();
        for (int t = threadIdx.x; t < kCnCols * ROWS; t += kCnThreads) {
            const int col = t / ROWS, row = t % ROWS, m1 = cs - 1 + kCnCols * g + col, m2 = d0 - 1 + row;
            bool small = false;
            if (row >= 1 && m1 >= cs && m1 < cs + P.ncol && m1 < P.nx && m2 < P.ny) {
                // cells (m1, m2), (m1, m2 - 1), (m1 - 1, m2), (m1 - 1, m2 - 1): corners 0..3
                const double *c0 = &M.v[0][col + 1][row], *c1 = c0 - 1, *c2 = c0 - ROWS, *c3 = c2 - 1;
                double Sv[NodeVals<NT>::N];
                double w1 = 0.0;
#pragma unroll
                for (int k = 0; k <= NT; k++) {
                    const int at = 4 * k * CS;
                    const double w = 0.25 * ((corner4<0>(c0 + at, CS) + corner4<1>(c1 + at, CS)) +
                                             (corner4<2>(c2 + at, CS) + corner4<3>(c3 + at, CS)));
                    if (k < NT) {
                        Sv[k] = w;
                        if ((P.mob >> k) & 1u) w1 += w;
                    } else {
                        Sv[NT + 1] = w;  // T
                    }
                }
                Sv[NT] = w1;
                Sv[NT + 2] = (c0[C::NU * CS] + c1[(C::NU + 1) * CS]) + (c2[(C::NU + 2) * CS] + c3[(C::NU + 3) * CS]);
                Sv[NT + 3] = (c0[C::WNU * CS] + c1[(C::WNU + 1) * CS]) + (c2[(C::WNU + 2) * CS] + c3[(C::WNU + 3) * CS]);
                Sv[NT + 4] = c3[C::ND * CS];
                Sv[NT + 5] = c3[C::WND * CS];
                small = node_finish<NT>(P, Q, m1, m2, Sv, vmin, vmax, any);
            }
            // the warp's nodes with small sums, one after the other
            for (unsigned f = __ballot_sync(0xffffffffu, small); f; f &= f - 1) {
                const int from = __ffs(f) - 1;
                ViscRange r{0.0, 0.0, 0};
                node_guard<NT>(P, __shfl_sync(0xffffffffu, m1, from), __shfl_sync(0xffffffffu, m2, from), &r);
                if (r.any) {
                    vmin = any ? fmin(vmin, r.lo) : r.lo;
                    vmax = any ? fmax(vmax, r.hi) : r.hi;
                    any = 1;
                }
            }
        }
        if (g + 1 == groups) break;
        // the last column becomes the next group's column 0
        double keep[(C::N * ROWS + kCnThreads - 1) / kCnThreads];
#pragma unroll
        for (int k = 0; k < (C::N * ROWS + kCnThreads - 1) / kCnThreads; k++) {
            const int t = k * kCnThreads + threadIdx.x;
            if (t < C::N * ROWS) keep[k] = M.v[t / ROWS][kCnCols][t % ROWS];
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < (C::N * ROWS + kCnThreads - 1) / kCnThreads; k++) {
            const int t = k * kCnThreads + threadIdx.x;
            if (t < C::N * ROWS) M.v[t / ROWS][0][t % ROWS] = keep[k];
        }
    }
    fold_minmax(vmin, vmax, any, P.ctr, owned, P.navg);
}

// Start of a fused averaging call: the call's counters, and the work k_move_fused left
// for it (first: not done by an earlier call on the same records): the sticky-air
// temperature resets, and the markers it kept a place for, whose viscosity comes
// from the rheology at the new position (allintere + viscalc, markmart.c:281,
// 320-332) into their records' log-viscosity and the call's |log-viscosity| bound.
template <bool MIXED>
__global__ void __launch_bounds__(256) k_fused_begin(const __grid_constant__ GridView G,
                                                     const __grid_constant__ MarkerView M,
                                                     const DevTypes *__restrict__ Ty,
                                                     const __grid_constant__ FusedMove F, int32_t first,
                                                     unsigned long long *navg)
{
    allow_next();
    wait_previous();
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        F.ctr->any = 0;
        F.ctr->kmin = ~0ull;
        F.ctr->kmax = 0ull;
        if (navg) *navg = 0ull;  // k_cellnodes counts the averaged markers
    }
    if (!first) return;
    const int32_t resets = F.ctr->ntreset, m = F.ctr->ndefer;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x, q0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (int64_t q = q0; q < resets; q += stride) M.T[F.treset[q]] = F.avg.tmp_ambient;
    if (m == 0) return;
    AvgArgsK V = F.avg;  // viscalc's impact weakening reads timesum (markmart.c:1886-1889)
    if (F.stepc) V.timesum = F.stepc[4 * *F.stepi];
    for (int64_t q = q0; q < m; q += stride) {
        const int2 d = F.defer[q];
        const int64_t i = d.x;
        const double x = M.x[i], y = M.y[i];
        const int mt = M.type[i];
        const double mtk = mt < 2 ? V.tmp_ambient : M.T[i];
        double pr = 0.0, mga = 0.0, mnu = 0.0;
        int64_t m10, m20;
        pressure_visc<MIXED>(G, Ty->t, V, x, y, mtk, M.hi ? M.hi[i] : 0.0, mt, false, true, pr, mga, mnu, m10, m20);
        const double lnu = record_lnu(G, V, x, y, mnu);
        if (d.y >= 0) {
            F.ra[d.y] = rec_with_lnu(F.ra[d.y], lnu);
        } else {
            OvfRec &r = F.ovf[-d.y - 1];
            r.a = rec_with_lnu(r.a, lnu);
        }
        atomicMax(&F.ctr->part[q % kFusedParts][2], __float_as_uint(__double2float_ru(fabs(lnu))));
    }
}

// movemark's counters and bucket counts to zero, as a kernel so that the launches of a
// run of steps overlap at this boundary too (a memset waits for and holds up both sides)
static __global__ void __launch_bounds__(256) k_fused_zero(uint4 *p, int64_t n)
{
    allow_next();
    wait_previous();
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) p[i] = make_uint4(0, 0, 0, 0);
}

// marktmax (markmart.c:354-360) on a fused averaging call
static __global__ void k_fused_tmax(const __grid_constant__ GridView G, const __grid_constant__ MarkerView M,
                             const __grid_constant__ AvgArgsK V)
{
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < M.n; i += stride) {
        const double x = M.x[i], y = M.y[i], Tm = M.T[i];
        const int mt = M.type[i];
        if (!(x > 0 && y > 0 && x < G.xsize && y < G.ysize && Tm > 0 && mt < kAvgTypes)) continue;
        if (V.gridmod > 1 && (M.id[i] % V.gridmod) != 0) continue;
        if (mt == 0) continue;
        const double mtk = mt < 2 ? V.tmp_ambient : Tm;
        if (M.tmax[i] < mtk) M.tmax[i] = mtk;
    }
}

// the contrast clamp (markmart.c:995-1009) from the call's viscosity range
static __global__ void __launch_bounds__(256) k_fused_clamp(int64_t nn, const FusedCounters *ctr, double nucontr,
                                                     double *nu, double *nd, double *stats)
{
    allow_next();
    wait_previous();
    double numin = 0.0, numax = 0.0;
    if (ctr->any) {
        numin = okey_inv(ctr->kmin);
        numax = okey_inv(ctr->kmax);
    }
    if (nucontr >= 1.0) numax = numin * nucontr; else numin = numax * nucontr;
    if (blockIdx.x == 0 && threadIdx.x == 0 && stats) {
        stats[0] = numin;
        stats[1] = numax;
    }
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t m3 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; m3 < nn; m3 += stride) {
        double v = nu[m3], u = v;
        const double w = nd[m3];
        if (u < numin) u = numin;
        if (u > numax) u = numax;
        if (u != v) nu[m3] = u;
        v = u = w;
        if (u < numin) u = numin;
        if (u > numax) u = numax;
        if (u != v) nd[m3] = u;
    }
}

}  // namespace i2g
