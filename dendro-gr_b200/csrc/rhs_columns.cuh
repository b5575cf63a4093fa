// Derivative pass of the split right-hand side: one thread per (x, y) column
// of a brick and variable, marching along z through the whole block.
//
// A CTA takes a brick of one block (BX x BY columns at most, every z) and a
// group of variables of one kind (with or without second derivatives), and
// stages one z plane of each (brick + 3-point halo) at a time into a ring of
// seven shared-memory slots with cp.async, three planes ahead.  When plane k
// has arrived a thread
//   * forms d/dx, d/dy (on halo planes too, where mixed derivatives need
//     them) and on the brick's planes d2/dx2, d2/dy2 and the x and y
//     dissipation from the plane in shared memory,
//   * keeps d/dx and d/dy in seven-plane rings in shared memory, and takes
//     d/dy of its neighbours' d/dx one plane later,
//   * completes the zone three planes back along z from the last seven values
//     of the variable (registers) and of its own d/dx and d/dy (rings).
// The plane loop is unrolled by seven, the length of every window, so ring
// slots and shared-memory addresses are constants and the register window
// rotates by name.
//
// Every stencil keeps the reference's order of rounded products and sums
// (rhs_brick.cuh).  Columns next to a physical x or y face are packed into
// warps of their own, which run a rolled loop with the table-driven
// one-sided closures and meet the others at the same barriers; next to a
// physical z face a pass after the march redoes three zones.
//
// What bounds it: the barrier per plane and shared-memory and FP64 issue
// (barrier 3-5 of 9-12 stall cycles per issue, LSU data pipe 34-47 % and FP64 17-22 %
// on a step of 477 mixed blocks, DRAM 20 %).  32 zones of a variable cost 102
// (55^3) to 119 (19^3) FP64 warp instructions and 35 to 45 shared loads; the
// form that this replaces (a cube of brick
// + halo per variable, one thread per zone, mixed derivatives through a
// cooperative halo pass, closures by per-term constant tables) issued about
// 430 instructions with 52 shared loads.  Derivative passes of one RK4 step:
// 19.8 M zones in 4,108 mixed blocks 58.2 -> 39 ms, a 2,708-block level mesh
// 9.3 -> 7.2 ms.  On 13^3 blocks, where a thread marches thirteen planes for
// seven, it gained on boundary blocks only and lost 16-31 % of the padded pass
// elsewhere; they run a form of their own (rhs_cube.cuh).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "bssn_common.cuh"
#include "rhs_brick.cuh"
#include "rhs_fused.cuh"

namespace bssn {
namespace {

// Scratch slots per zone (in pairs, so both passes move 16 bytes): with
// second derivatives dx dy | xx yy | dz zz | xz yz | xy ko, without
// dx dy | dz ko.  A variable's pairs appear in the order in which the
// column pass completes them.
constexpr int kPairsSecond = 5, kPairsFirst = 2;
constexpr int kSecondVars = 11, kFirstVars = 13;
static_assert(2 * (kSecondVars * kPairsSecond + kFirstVars * kPairsFirst) == kSplitSlots, "scratch slots");

// visiting position (stage_order) of the i-th variable with / without second
// derivatives, and the first scratch pair of a position
__host__ __device__ constexpr int second_step(int i) { return i < 9 ? i : i + 3; }
__host__ __device__ constexpr int first_step(int i) { return i < 3 ? i + 9 : i + 11; }
__host__ __device__ constexpr int pair_base(int step) {
    return step < 9 ? kPairsSecond * step
         : step < 12 ? 9 * kPairsSecond + kPairsFirst * (step - 9)
         : step < 14 ? 9 * kPairsSecond + 3 * kPairsFirst + kPairsSecond * (step - 12)
         : kSecondVars * kPairsSecond + 3 * kPairsFirst + kPairsFirst * (step - 14);
}

// Shape of a brick's columns: rows BX x BY; V2 / V1 variables with / without
// second derivatives per CTA of T threads (as many columns as MAXT holds, at
// most ITER staged points a thread, the groups of a kind evened out).
constexpr int kColRing = 7;   // slots of every ring, planes per unrolled turn
constexpr int kColAhead = 3;  // planes in flight

template <int BX_, int BY_>
struct ColShape {
    static constexpr int BX = BX_, BY = BY_;
    static constexpr int TX = BX + 2 * PW, TY = BY + 2 * PW;
    static constexpr int COLS = BX * BY;
    static constexpr int PL = TX * TY;   // staged points of a plane
    static constexpr int DXP = BX * TY;  // d/dx of a plane, with the halo rows
    // Two CTAs of at most 256 threads per SM (31^3: 256 at 128 registers, 19^3:
    // 192 at 160), or, for full-width strips of 55^3 blocks, whose halo rows weigh more than a second CTA
    // gives, one of 512: derivative passes of one RK4 step on 98 such blocks
    // (10.8 M zones) 21.5 ms with 49 x 10 columns, 24.1 with 49 x 13 in 640
    // threads, 26.7 with two CTAs of 49 x 5.  ITER, the staged points whose
    // pointers a thread keeps, has not been swept.
    static constexpr int MAXT = BX >= 49 ? 512 : 256;
    static constexpr int MINB = BX >= 49 ? 1 : 2;
    static constexpr int ITER = BX >= 9 ? 3 : 4;
    static constexpr int threads(int v) {
        const int need = v * COLS > (v * PL + ITER - 1) / ITER ? v * COLS : (v * PL + ITER - 1) / ITER;
        return (need + 31) / 32 * 32;
    }
    static constexpr int groups(int vars) {
        int v = vars;
        while (v > 1 && threads(v) > MAXT) v--;
        return (vars + v - 1) / v;
    }
    static constexpr int G2 = groups(kSecondVars), G1 = groups(kFirstVars);
    static constexpr int V2 = (kSecondVars + G2 - 1) / G2, V1 = (kFirstVars + G1 - 1) / G1;
    static constexpr int T = threads(V2 > V1 ? V2 : V1);
    // points of d/dx on the halo rows per thread
    static constexpr int HIT = (V2 * 2 * PW * BX + T - 1) / T;
    static constexpr int SMEM2 = kColRing * V2 * (PL + DXP + COLS), SMEM1 = kColRing * V1 * PL;
    static constexpr size_t SMEM = sizeof(double) * (SMEM2 > SMEM1 ? SMEM2 : SMEM1);
    static_assert(T <= MAXT && SMEM <= 224 * 1024, "a CTA's threads and shared memory");
};

// x / d for 0 <= x < 2^15 (rounded down) from r = 1 / d: x + 1/2 stays at
// least 1 / (2 d) away from every multiple of d, far more than the rounding.
__device__ __forceinline__ int div_small(int x, float r) { return (int)(((float)x + 0.5f) * r); }

template <int N>
__device__ __forceinline__ double fold6(const double (&c)[N], const double (&u)[6], const int (&p)[N]) {
    double t = __dmul_rn(c[0], u[p[0]]);
#pragma unroll
    for (int q = 1; q < N; q++) t = __dadd_rn(t, __dmul_rn(c[q], u[p[q]]));
    return t;
}

// weights of the first-derivative closures along z, zones next to the face
// in increasing z, over the five points they use in increasing z
__constant__ double kZCloD1[2][3][5] = {
    {{-25, 48, -36, 16, -3}, {-3, -10, 18, -6, 1}, {1, -8, 0, 8, -1}},
    {{1, -8, 0, 8, -1}, {-1, 6, -18, 10, 3}, {3, -16, 36, -48, 25}}};

// One-sided closures along a line that ends at a physical face, from its six
// points next to the face.
__device__ __forceinline__ void z_closures_d1(bool lo, const double (&u)[6], const AxisCoef& cf, double d1[3]) {
    if (lo) {
        { const double c[5] = {-25, 48, -36, 16, -3}; const int p[5] = {0, 1, 2, 3, 4}; d1[0] = fold6(c, u, p); }
        { const double c[5] = {-3, -10, 18, -6, 1}; const int p[5] = {0, 1, 2, 3, 4}; d1[1] = fold6(c, u, p); }
        { const double c[4] = {1, -8, 8, -1}; const int p[4] = {0, 1, 3, 4}; d1[2] = fold6(c, u, p); }
    } else {
        { const double c[4] = {1, -8, 8, -1}; const int p[4] = {1, 2, 4, 5}; d1[0] = fold6(c, u, p); }
        { const double c[5] = {-1, 6, -18, 10, 3}; const int p[5] = {1, 2, 3, 4, 5}; d1[1] = fold6(c, u, p); }
        { const double c[5] = {3, -16, 36, -48, 25}; const int p[5] = {1, 2, 3, 4, 5}; d1[2] = fold6(c, u, p); }
    }
#pragma unroll
    for (int q = 0; q < 3; q++) d1[q] = __dmul_rn(d1[q], cf.ih12);
}
__device__ __forceinline__ void z_closures(bool lo, const double (&u)[6], const AxisCoef& cf, double d1[3],
                                           double d2[3], double ko[3]) {
    z_closures_d1(lo, u, cf, d1);
    if (lo) {
        { const double c[6] = {45, -154, 214, -156, 61, -10}; const int p[6] = {0, 1, 2, 3, 4, 5}; d2[0] = fold6(c, u, p); }
        { const double c[6] = {10, -15, -4, 14, -6, 1}; const int p[6] = {0, 1, 2, 3, 4, 5}; d2[1] = fold6(c, u, p); }
        { const double c[5] = {-1, 16, -30, 16, -1}; const int p[5] = {0, 1, 2, 3, 4}; d2[2] = fold6(c, u, p); }
        { const double c[4] = {1, -3, 3, -1}; const int p[4] = {3, 2, 1, 0}; ko[0] = fold6(c, u, p); }
        { const double c[5] = {1, -6, 12, -10, 3}; const int p[5] = {4, 3, 2, 1, 0}; ko[1] = fold6(c, u, p); }
        { const double c[6] = {1, -6, 15, -19, 12, -3}; const int p[6] = {5, 4, 3, 2, 1, 0}; ko[2] = fold6(c, u, p); }
    } else {
        { const double c[5] = {-1, 16, -30, 16, -1}; const int p[5] = {1, 2, 3, 4, 5}; d2[0] = fold6(c, u, p); }
        { const double c[6] = {1, -6, 14, -4, -15, 10}; const int p[6] = {0, 1, 2, 3, 4, 5}; d2[1] = fold6(c, u, p); }
        { const double c[6] = {-10, 61, -156, 214, -154, 45}; const int p[6] = {0, 1, 2, 3, 4, 5}; d2[2] = fold6(c, u, p); }
        { const double c[6] = {1, -6, 15, -19, 12, -3}; const int p[6] = {0, 1, 2, 3, 4, 5}; ko[0] = fold6(c, u, p); }
        { const double c[5] = {1, -6, 12, -10, 3}; const int p[5] = {1, 2, 3, 4, 5}; ko[1] = fold6(c, u, p); }
        { const double c[4] = {1, -3, 3, -1}; const int p[4] = {2, 3, 4, 5}; ko[2] = fold6(c, u, p); }
    }
#pragma unroll
    for (int q = 0; q < 3; q++) {
        const int cs = lo ? q : 3 + q;
        d2[q] = __dmul_rn(d2[q], cf.ih2_12);
        ko[q] = __ddiv_rn(ko[q], closure_smr(cs, cf));
    }
}

template <int N>
__device__ __forceinline__ void col_wait_pending() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

// Extents of the zones a brick's passes cover: all of them, or, when the
// right-hand side goes to the zipped grid (g.gx > 0), only the zones owning
// their node (a node on a block's upper face belongs to the next block
// unless the face lies on the grid's upper boundary: the zip's owner rule).
// keep_faces: layers on a physical face stay whoever owns them (one-sided
// closures of the next layers use their derivatives).
__device__ __forceinline__ void owned_extent(const BssnBlockDesc& blk, const BrickTask& tk, const ZipGrid& g,
                                             bool keep_faces, int ex[3]) {
    const int n = blk.sz - 2 * PW;
    const int gd[3] = {g.gx, g.gy, g.gz};
#pragma unroll
    for (int d = 0; d < 3; d++) {
        ex[d] = tk.e[d];
        if (g.drop && tk.o[d] + ex[d] == n && (g.drop[tk.blk] >> d & 1)) ex[d]--;
        if (g.gx && tk.o[d] + ex[d] == n && blk.g0[d] + n - 1 != gd[d] - 1 &&
            !(keep_faces && (blk.bflag & (2u << (2 * d)))))
            ex[d]--;
    }
}

// All warps of the CTA, which run two versions of the plane loop with the
// same number of barriers.
__device__ __forceinline__ void col_barrier() { asm volatile("bar.sync 0;\n" ::: "memory"); }

template <bool SECOND, class Sh, bool ZIP>
__device__ __forceinline__ void column_march(const uint8_t* steps, int nv, const BrickTask& tk, const BssnBlockDesc& blk,
                                             const int ex[3], const double* const* src, const AxisCoef* cfs,
                                             const ClosureTables& CT, double* __restrict__ S, int64_t zs,
                                             const ZipGrid& g, double* ring) {
    constexpr int BX = Sh::BX, TX = Sh::TX, T = Sh::T, PL = Sh::PL, COLS = Sh::COLS;
    constexpr int V = SECOND ? Sh::V2 : Sh::V1;
    constexpr int RS = V * PL;                               // ring slot
    constexpr int DX7 = V * Sh::DXP, DY7 = V * COLS;
    double* dxs = ring + kColRing * RS;   // [7][V][TY][BX]: d/dx
    double* dys = dxs + kColRing * DX7;   // [7][V][BY][BX]: d/dy
    const int tid = threadIdx.x;
    const int s = blk.sz;
    const int o0 = tk.o[0], o1 = tk.o[1];
    const int np = ex[2] + 2 * PW;  // planes staged
    auto step_of = [&](int v) { return (int)steps[v]; };  // visiting position of the group's v-th variable

    // staged points of this thread: source pointer at the first plane and
    // place in a ring slot (-1: none, <= -2: outside the grid, zero)
    constexpr int ITER = (V * PL + T - 1) / T;
    const int sx = ex[0] + 2 * PW, pts = sx * (ex[1] + 2 * PW);
    const float rsx = 1.0f / sx, rpts = 1.0f / pts;
    const int64_t zst = ZIP ? (int64_t)g.gx * g.gy : (int64_t)s * s;
    const double* sp[ITER];
    int sd[ITER];
#pragma unroll
    for (int q = 0; q < ITER; q++) {
        const int idx = tid + q * T;
        sd[q] = -1;
        sp[q] = nullptr;
        if (idx < nv * pts) {
            const int v = div_small(idx, rpts), r = idx - v * pts, y = div_small(r, rsx), x = r - y * sx;
            const int place = v * PL + y * TX + x;
            const double* base = src[step_of(v)];
            if (!ZIP) {
                sp[q] = base + (o0 + x) + (int64_t)s * (o1 + y);
                sd[q] = place;
            } else {  // padded coordinate c is node g0 + c - 3
                const int X = blk.g0[0] + o0 + x - PW, Y = blk.g0[1] + o1 + y - PW;
                const bool in = X >= 0 && Y >= 0 && X < g.gx && Y < g.gy;
                sp[q] = base + (in ? X + (int64_t)g.gx * Y : 0) + zst * (blk.g0[2] - PW);
                sd[q] = in ? place : -2 - place;
            }
        }
    }
    const int z0 = ZIP ? blk.g0[2] - PW : 0;  // node plane of plane 0
    auto stage = [&](int k, double* dst) {
        if (k < np) {
            const bool zin = !ZIP || (z0 + k >= 0 && z0 + k < g.gz);
#pragma unroll
            for (int q = 0; q < ITER; q++) {
                if (sd[q] >= 0 && zin)
                    cp_async8(dst + sd[q], sp[q]);
                else if (ZIP && sd[q] != -1)
                    dst[sd[q] >= 0 ? sd[q] : -2 - sd[q]] = 0.0;
                sp[q] += zst;
            }
        }
        cp_async_commit();
    };

    // this thread's column: the columns away from physical x and y faces
    // first (of every variable), then those next to a y face, then those next
    // to an x face only
    const unsigned bf = blk.bflag;
    auto near_lo = [&](int o, bool face) { return face ? max(0, 3 - o) : 0; };
    auto near_hi = [&](int o, int e, bool face) { return face ? max(0, o + e - (s - 9)) : 0; };
    const int nlx = near_lo(o0, bf & 1u), nx = nlx + near_hi(o0, ex[0], bf & 2u), wx = ex[0] - nx;
    const int nly = near_lo(o1, bf & 4u), ny = nly + near_hi(o1, ex[1], bf & 8u), hy = ex[1] - ny;
    int v, cx, cy;
    bool active = true;
    {
        int c = tid;
        const int inner = wx * hy, rows = ex[0] * ny, strips = nx * hy;
        if (c < nv * inner) {
            v = div_small(c, 1.0f / inner);
            c -= v * inner;
            cy = div_small(c, 1.0f / wx);
            cx = nlx + c - cy * wx;
            cy += nly;
        } else if ((c -= nv * inner) < nv * rows) {
            v = div_small(c, 1.0f / rows);
            c -= v * rows;
            cy = div_small(c, 1.0f / ex[0]);
            cx = c - cy * ex[0];
            if (cy >= nly) cy += hy;
        } else if ((c -= nv * rows) < nv * strips) {
            v = div_small(c, 1.0f / strips);
            c -= v * strips;
            cy = div_small(c, 1.0f / nx);
            cx = c - cy * nx;
            cy += nly;
            if (cx >= nlx) cx += wx;
        } else {
            active = false;
            v = cx = cy = 0;
        }
    }
    const int ax = o0 + PW + cx, ay = o1 + PW + cy;  // padded coordinates
    const int toff = v * PL + (cy + PW) * TX + cx + PW;
    const int mx = v * Sh::DXP + (cy + PW) * BX + cx, my = v * COLS + cy * BX + cx;
    double2* const w0 = reinterpret_cast<double2*>(S) + (int64_t)pair_base(active ? step_of(v) : 0) * zs + (cx + BX * cy);
    // d/dx on the halo rows of the brick's planes
    constexpr int HIT = Sh::HIT;
    int ht[HIT], hd[HIT], ha[HIT];
    if (SECOND) {
#pragma unroll
        for (int q = 0; q < HIT; q++) {
            const int idx = tid + q * T;
            ht[q] = -1;
            hd[q] = ha[q] = 0;
            if (idx < nv * 2 * PW * ex[0]) {
                const int hv = div_small(idx, 1.0f / (2 * PW * ex[0])), r = idx - hv * 2 * PW * ex[0];
                const int h = div_small(r, 1.0f / ex[0]), i = r - h * ex[0];
                const int row = h < PW ? h : ex[1] + h;
                ht[q] = hv * PL + row * TX + i + PW;
                hd[q] = hv * Sh::DXP + row * BX + i;
                const int a = o0 + PW + i;
                ha[q] = near_face(a, s, bf & 1u, bf & 2u) ? a : 0;  // padded x next to a face
            }
        }
    }
    auto halo_rows = [&](const double* cur, double* dxk) {
#pragma unroll
        for (int q = 0; q < HIT; q++) {
            if (ht[q] >= 0) {
                const double* t = cur + ht[q];
                double dx = d1_in(t, 1, cfs[0]);
                if (ha[q]) {
                    const int cs = closure_case(ha[q], s, bf & 1u);
                    dx = __dmul_rn(closure_tab(CT, 0, cs, t + (cs < 3 ? 3 : s - 9) - ha[q], 1), cfs[0].ih12);
                }
                dxk[hd[q]] = dx;
            }
        }
    };
    // zones whose z dissipation is added after the march: next to a lower /
    // upper physical z face
    auto z_near = [&](int k) { return ((bf & 16u) && k <= 5) || ((bf & 32u) && k >= s - 6); };

#pragma unroll
    for (int k = 0; k < kColAhead; k++) stage(k, ring + k * RS);

    if (!__any_sync(0xffffffffu, active && (near_face(ax, s, bf & 1u, bf & 2u) || near_face(ay, s, bf & 4u, bf & 8u)))) {
        // no column next to a physical x or y face in this warp
        double uw[7], kxy[7], xyq[7];
        double2* w = w0 - PW * COLS;  // zone of plane kb (lead), plane by plane
#pragma unroll 1
        for (int kb = 0; kb < np; kb += kColRing) {
#pragma unroll
            for (int p = 0; p < kColRing; p++) {
                const int k = kb + p;
                if (k < np) {
                    col_wait_pending<kColAhead - 1>();
                    col_barrier();  // plane k complete; the slot staged next was read at plane k - 4
                    stage(k + kColAhead, ring + (p + kColAhead) % kColRing * RS);
                    const bool brick = k >= PW && k < np - PW;  // a plane of the brick
                    const double* cur = ring + p * RS;
                    if (active) {
                        const double* t = cur + toff;
                        uw[p] = t[0];
                        if (SECOND && k >= PW + 1 && k <= np - PW)  // d/dy of d/dx on plane k - 1
                            xyq[(p + 6) % 7] = d1_fast_in(dxs + (p + 6) % 7 * DX7 + mx, BX, cfs[1]);
                        double dx = 0.0, dy = 0.0;
                        if (SECOND || brick) {
                            double tx[7], ty[7];
#pragma unroll
                            for (int q = 0; q < 7; q++) {
                                tx[q] = q == 3 ? uw[p] : t[q - 3];
                                ty[q] = q == 3 ? uw[p] : t[(q - 3) * TX];
                            }
                            dx = d1_in(tx + 3, 1, cfs[0]);
                            dy = d1_in(ty + 3, 1, cfs[1]);
                            if (SECOND) {
                                dxs[p * DX7 + mx] = dx;
                                dys[p * DY7 + my] = dy;
                            }
                            if (brick) {
                                w[p * COLS] = make_double2(dx, dy);
                                kxy[p] = ko_in(tx + 3, 1, cfs[0]) + ko_in(ty + 3, 1, cfs[1]);
                                if (SECOND)
                                    w[p * COLS + zs] = make_double2(d2_in(tx + 3, 1, cfs[0]), d2_in(ty + 3, 1, cfs[1]));
                            }
                        }
                        if (k >= 2 * PW) {  // the zone of plane k - 3
                            double win[7];
#pragma unroll
                            for (int q = 0; q < 7; q++) win[q] = uw[(p + 1 + q) % 7];
                            const double dz = d1_in(win + 3, 1, cfs[2]);
                            const double kz = ko_in(win + 3, 1, cfs[2]);
                            const double kk = kxy[(p + 4) % 7];
                            const double ko = z_near(k - PW) ? kk : kk + kz;
                            double2* wl = w + (p - PW) * COLS;
                            if (SECOND) {
                                double ox[7], oy[7];  // own d/dx, d/dy of planes k - 6 .. k
#pragma unroll
                                for (int q = 0; q < 7; q++) {
                                    ox[q] = q == 3 ? 0.0 : q == 6 ? dx : dxs[(p + 1 + q) % 7 * DX7 + mx];
                                    oy[q] = q == 3 ? 0.0 : q == 6 ? dy : dys[(p + 1 + q) % 7 * DY7 + my];
                                }
                                wl[2 * zs] = make_double2(dz, d2_in(win + 3, 1, cfs[2]));
                                wl[3 * zs] = make_double2(d1_fast_in(ox + 3, 1, cfs[2]), d1_fast_in(oy + 3, 1, cfs[2]));
                                wl[4 * zs] = make_double2(xyq[(p + 4) % 7], ko);
                            } else {
                                wl[zs] = make_double2(dz, ko);
                            }
                        }
                    }
                    if (SECOND && brick) halo_rows(cur, dxs + p * DX7);
                }
            }
            w += kColRing * COLS;
        }
    } else {
        // the same with one-sided closures, one plane at a time: windows
        // shifted by moves, ring slots computed
        const int cxc = near_face(ax, s, bf & 1u, bf & 2u) ? closure_case(ax, s, bf & 1u) : -1;
        const int cyc = near_face(ay, s, bf & 4u, bf & 8u) ? closure_case(ay, s, bf & 4u) : -1;
        // the first of the six points next to the face, relative to the column
        const int fx = (cxc < 3 ? 3 : s - 9) - ax, fy = (cyc < 3 ? 3 : s - 9) - ay;
        double uw[7], kxy[4], xyq[3];
#pragma unroll
        for (int q = 0; q < 7; q++) uw[q] = 0.0;
        kxy[0] = kxy[1] = kxy[2] = kxy[3] = xyq[0] = xyq[1] = xyq[2] = 0.0;
        double2* w = w0 - PW * COLS;  // zone of plane k
        int r7 = 0;                   // ring slot of plane k
        auto slot = [&](int j) { return r7 >= j ? r7 - j : r7 - j + kColRing; };  // of plane k - j
#pragma unroll 1
        for (int k = 0; k < np; k++) {
            col_wait_pending<kColAhead - 1>();
            col_barrier();
            stage(k + kColAhead, ring + slot(kColRing - kColAhead) * RS);
            const bool brick = k >= PW && k < np - PW;
            const double* cur = ring + r7 * RS;
            if (active) {
                const double* t = cur + toff;
#pragma unroll
                for (int q = 0; q < 6; q++) uw[q] = uw[q + 1];
                uw[6] = t[0];
#pragma unroll
                for (int q = 0; q < 3; q++) kxy[q] = kxy[q + 1];
                xyq[0] = xyq[1];
                xyq[1] = xyq[2];
                if (SECOND && k >= PW + 1 && k <= np - PW) {
                    const double* m = dxs + slot(1) * DX7 + mx;
                    xyq[2] = d1_fast_in(m, BX, cfs[1]);
                    if (cyc >= 0) xyq[2] = __dmul_rn(closure_tab(CT, 0, cyc, m + fy * BX, BX), cfs[1].ih12);
                }
                double dx = 0.0, dy = 0.0;
                if (SECOND || brick) {
                    dx = d1_in(t, 1, cfs[0]);
                    dy = d1_in(t, TX, cfs[1]);
                    if (cxc >= 0) dx = __dmul_rn(closure_tab(CT, 0, cxc, t + fx, 1), cfs[0].ih12);
                    if (cyc >= 0) dy = __dmul_rn(closure_tab(CT, 0, cyc, t + fy * TX, TX), cfs[1].ih12);
                    if (SECOND) {
                        dxs[r7 * DX7 + mx] = dx;
                        dys[r7 * DY7 + my] = dy;
                    }
                    if (brick) {
                        w[0] = make_double2(dx, dy);
                        double kx = ko_in(t, 1, cfs[0]), ky = ko_in(t, TX, cfs[1]);
                        if (cxc >= 0) kx = __ddiv_rn(closure_tab(CT, 2, cxc, t + fx, 1), closure_smr(cxc, cfs[0]));
                        if (cyc >= 0) ky = __ddiv_rn(closure_tab(CT, 2, cyc, t + fy * TX, TX), closure_smr(cyc, cfs[1]));
                        kxy[3] = kx + ky;
                        if (SECOND) {
                            double xx = d2_in(t, 1, cfs[0]), yy = d2_in(t, TX, cfs[1]);
                            if (cxc >= 0) xx = __dmul_rn(closure_tab(CT, 1, cxc, t + fx, 1), cfs[0].ih2_12);
                            if (cyc >= 0) yy = __dmul_rn(closure_tab(CT, 1, cyc, t + fy * TX, TX), cfs[1].ih2_12);
                            w[zs] = make_double2(xx, yy);
                        }
                    }
                }
                if (k >= 2 * PW) {
                    const double dz = d1_in(uw + 3, 1, cfs[2]);
                    const double kz = ko_in(uw + 3, 1, cfs[2]);
                    const double ko = z_near(k - PW) ? kxy[0] : kxy[0] + kz;
                    double2* wl = w - PW * COLS;
                    if (SECOND) {
                        double ox[7], oy[7];
#pragma unroll
                        for (int q = 0; q < 7; q++) {
                            ox[q] = q == 3 ? 0.0 : q == 6 ? dx : dxs[slot(6 - q) * DX7 + mx];
                            oy[q] = q == 3 ? 0.0 : q == 6 ? dy : dys[slot(6 - q) * DY7 + my];
                        }
                        wl[2 * zs] = make_double2(dz, d2_in(uw + 3, 1, cfs[2]));
                        wl[3 * zs] = make_double2(d1_fast_in(ox + 3, 1, cfs[2]), d1_fast_in(oy + 3, 1, cfs[2]));
                        wl[4 * zs] = make_double2(xyq[0], ko);
                    } else {
                        wl[zs] = make_double2(dz, ko);
                    }
                }
            }
            if (SECOND && brick) halo_rows(cur, dxs + r7 * DX7);
            r7 = r7 == kColRing - 1 ? 0 : r7 + 1;
            w += COLS;
        }
    }

    // The three zones next to a physical z face: everything along z again,
    // one-sided.  The variable's six points come from global memory, d/dx,
    // d/dy, xy and the x and y dissipation back from the scratch, where this
    // thread wrote them.
    if (!active || !(bf & 48u)) return;
#pragma unroll 1
    for (int side = 0; side < 2; side++) {
        const bool lo = side == 0;
        if (!(bf & (lo ? 16u : 32u))) continue;
        const int f = lo ? 3 : s - 9;         // first of the six points
        const int q0 = lo ? 0 : s - 6 - PW;   // first of the three zones
        const double* base = src[step_of(v)];
        double u[6], dz[3], zz[3], kz[3], xz[3], yz[3];
#pragma unroll
        for (int j = 0; j < 6; j++) {
            if (ZIP)
                u[j] = base[blk.g0[0] + ax - PW + (int64_t)g.gx * (blk.g0[1] + ay - PW) + zst * (blk.g0[2] + f + j - PW)];
            else
                u[j] = base[ax + (int64_t)s * ay + zst * (f + j)];
        }
        z_closures(lo, u, cfs[2], dz, zz, kz);
        if (SECOND) {
            const double2* wd = w0 + (int64_t)(f - PW + (lo ? 0 : 1)) * COLS;  // the five planes the closures use
#pragma unroll
            for (int q = 0; q < 3; q++) xz[q] = yz[q] = 0.0;
#pragma unroll 1
            for (int j = 0; j < 5; j++, wd += COLS) {
                const double2 dxy = *wd;
#pragma unroll
                for (int q = 0; q < 3; q++) {
                    const double cc = kZCloD1[side][q][j];
                    if (cc != 0.0) {
                        xz[q] = __dadd_rn(xz[q], __dmul_rn(cc, dxy.x));
                        yz[q] = __dadd_rn(yz[q], __dmul_rn(cc, dxy.y));
                    }
                }
            }
        }
#pragma unroll
        for (int q = 0; q < 3; q++) {
            double2* wz = w0 + (int64_t)(q0 + q) * COLS;
            if (SECOND) {
                wz[2 * zs] = make_double2(dz[q], zz[q]);
                wz[3 * zs] = make_double2(__dmul_rn(xz[q], cfs[2].ih12), __dmul_rn(yz[q], cfs[2].ih12));
                const double2 pk = wz[4 * zs];
                wz[4 * zs] = make_double2(pk.x, pk.y + kz[q]);
            } else {
                wz[zs] = make_double2(dz[q], wz[zs].y + kz[q]);
            }
        }
    }
}

__host__ __device__ constexpr int col_groups(int n, int v) { return (n + v - 1) / v; }

// A block given by value, for launches without a mesh.
struct SplitOne {
    BssnBlockDesc blk;
    AxisCoef axis[3];
};

// The q-th brick of such a block under bx x by columns.
__device__ __forceinline__ BrickTask one_brick(int side, int q, int bx, int by) {
    const int n = side - 2 * PW, nbx = (n + bx - 1) / bx;
    BrickTask tk;
    int o, e;
    tk.blk = 0;
    split1(n, bx, q % nbx, o, e);
    tk.o[0] = (int16_t)o;
    tk.e[0] = (int16_t)e;
    split1(n, by, q / nbx, o, e);
    tk.o[1] = (int16_t)o;
    tk.e[1] = (int16_t)e;
    tk.o[2] = 0;
    tk.e[2] = (int16_t)n;
    return tk;
}

// One CTA per (brick, group of variables): the groups with second derivatives
// first.
template <class Sh, bool ZIP>
__device__ __forceinline__ void column_cta(const ConstVars& u, const BrickTask& tk, const BssnBlockDesc& blk,
                                           const AxisCoef* axis, int task, int group, double* __restrict__ S,
                                           int64_t zs, const ZipGrid& g, int nz, const ColVars& vars) {
    extern __shared__ __align__(16) double smem[];
    __shared__ const double* src[NVARS];
    __shared__ AxisCoef cfs[3];
    __shared__ ClosureTables CT;
    __shared__ uint8_t steps[Sh::V2 > Sh::V1 ? Sh::V2 : Sh::V1];
    const int g2 = col_groups(vars.n2, Sh::V2);
    const int i0 = group < g2 ? group * Sh::V2 : (group - g2) * Sh::V1;  // the group's first variable
    const int nv = group < g2 ? min(Sh::V2, vars.n2 - i0) : min(Sh::V1, vars.n1 - i0);
    const int tid = threadIdx.x;
    if (tid < NVARS) src[tid] = u.p[stage_order(tid)] + (ZIP ? 0 : blk.offset);
    if (tid < nv) steps[tid] = group < g2 ? vars.second[i0 + tid] : vars.first[i0 + tid];
    if (tid < 24) (&cfs[0].ih60)[tid] = (&axis[0].ih60)[tid];
    if (blk.bflag & 15u) fill_closures(CT, tid);
    int ex[3];
    owned_extent(blk, tk, g, true, ex);
    __syncthreads();
    double* Sb = S + 2 * (int64_t)task * nz;
    if (group < g2)
        column_march<true, Sh, ZIP>(steps, nv, tk, blk, ex, src, cfs, CT, Sb, zs, g, smem);
    else
        column_march<false, Sh, ZIP>(steps, nv, tk, blk, ex, src, cfs, CT, Sb, zs, g, smem);
}

template <class Sh, bool ZIP>
__global__ void __launch_bounds__(Sh::T, Sh::MINB)
column_kernel(ConstVars u, const BssnBlockDesc* __restrict__ blocks, const AxisCoef* __restrict__ axis,
              const BrickTask* __restrict__ tasks, double* __restrict__ S, int64_t zs, ZipGrid g, int nz,
              ColVars vars) {
    const int groups = col_groups(vars.n2, Sh::V2) + col_groups(vars.n1, Sh::V1);
    const int task = blockIdx.x / groups;
    const BrickTask tk = tasks[task];
    const BssnBlockDesc blk = blocks[tk.blk];
    column_cta<Sh, ZIP>(u, tk, blk, axis + 3 * (int64_t)tk.blk, task, blockIdx.x % groups, S, zs, g, nz, vars);
}

// The bricks of one block.
template <class Sh>
__global__ void __launch_bounds__(Sh::T, Sh::MINB)
column_one_kernel(ConstVars u, const __grid_constant__ SplitOne one, double* __restrict__ S, int64_t zs, int nz,
                  ColVars vars) {
    const int groups = col_groups(vars.n2, Sh::V2) + col_groups(vars.n1, Sh::V1);
    const int task = blockIdx.x / groups;
    const BrickTask tk = one_brick(one.blk.sz, task, Sh::BX, Sh::BY);
    column_cta<Sh, false>(u, tk, one.blk, one.axis, task, blockIdx.x % groups, S, zs, ZipGrid{0, 0, 0}, nz, vars);
}

}  // namespace
}  // namespace bssn
