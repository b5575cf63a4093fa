// Derivative pass of 13^3 blocks: one CTA per block and variable, the padded
// cube in shared memory, one thread per line of points.
//
// The column pass (rhs_columns.cuh) stages thirteen planes for the seven of
// such a block, with a barrier and a CTA-wide wait at each.  Here the cube is
// fetched once and every derivative of a direction is formed by threads that
// hold a whole line of thirteen points along it in registers: thirteen shared
// loads for the first, second and dissipation derivatives of seven zones, and
// one-sided closures at fixed places of the line, the same for every thread of
// a group, so physical faces cost no divergence.  The three axes run the same
// code at different strides (each axis with code of its own spent a quarter of
// its time waiting for instructions).
//
// What bounds it: the latency of the fetch at 22 warps an SM (80 registers,
// 45 KB a CTA), FP64 30 % busy, half of the copy rate.  CTAs that run together
// take the same variable of neighbouring blocks, kCubeGroup blocks at a time:
// 1,728 blocks 338 us against 381 with a block's variables side by side, 8,000
// blocks 1.57 ms against 1.73, and 1.70 over all blocks at once.  Padded blocks
// without physical faces, derivative pass, against the column pass (and the
// cube form with a thread per zone before that): 1,728 blocks 335 us, 436 (372);
// 8,000 blocks 1.57 ms, 1.97 (1.64); 1,728 blocks with three faces each 369 us,
// 1,049 (1,042).  One RK4 step of 512 blocks from the node grid: 0.78 ms, 1.28.
#pragma once
#include "rhs_columns.cuh"

namespace bssn {
namespace {

// A CTA is three groups of 64 threads, one per axis, and takes one variable.
struct Cube {
    static constexpr int S = 13, N = 7, T = 192, ZONES = N * N * N;
    // Places in shared memory.  Planes lie eight banks (of 8 bytes) apart, so
    // that the fourteen lines of a half warp (seven along one axis, two along
    // the next) meet on no bank (along z on two): of the cube, of d/dx (13 rows
    // of 7), and of d/dy and single values of the zones (7 rows of 7).
    static constexpr int UP = 184, XP = 104, HP = 56;
    static constexpr int U = S * UP, DX = S * XP, DY = S * HP, Z = N * HP;
    static constexpr size_t SMEM = sizeof(double) * (U + DX + DY + 3 * Z);
};
// blocks whose CTAs of one variable are adjacent in the grid
constexpr int kCubeGroup = 1024;

// faces: bit 0 / 1, the line's lower / upper end lies on a physical face.
// FAST: the outer stage of a mixed derivative (multiply-adds).
template <bool FAST>
__device__ __forceinline__ void line_d1(const double (&r)[13], unsigned faces, const AxisCoef& cf, double d1[7]) {
#pragma unroll
    for (int i = 0; i < 7; i++) d1[i] = FAST ? d1_fast_in(r + PW + i, 1, cf) : d1_in(r + PW + i, 1, cf);
#pragma unroll
    for (int f = 0; f < 2; f++) {
        if (!(faces >> f & 1u)) continue;
        double u[6];
#pragma unroll
        for (int q = 0; q < 6; q++) u[q] = r[PW + f + q];
        z_closures_d1(f == 0, u, cf, d1 + 4 * f);
    }
}

// d2 only where `second`.
__device__ __forceinline__ void line_all(const double (&r)[13], unsigned faces, bool second, const AxisCoef& cf,
                                         double d1[7], double d2[7], double ko[7]) {
#pragma unroll
    for (int i = 0; i < 7; i++) {
        d1[i] = d1_in(r + PW + i, 1, cf);
        ko[i] = ko_in(r + PW + i, 1, cf);
        d2[i] = 0.0;
    }
    if (second)
#pragma unroll
        for (int i = 0; i < 7; i++) d2[i] = d2_in(r + PW + i, 1, cf);
#pragma unroll
    for (int f = 0; f < 2; f++) {
        if (!(faces >> f & 1u)) continue;
        double u[6];
#pragma unroll
        for (int q = 0; q < 6; q++) u[q] = r[PW + f + q];
        z_closures(f == 0, u, cf, d1 + 4 * f, d2 + 4 * f, ko + 4 * f);
    }
}

__device__ __forceinline__ void get_line(double (&r)[13], const double* u, int st) {
#pragma unroll
    for (int q = 0; q < 13; q++) r[q] = u[q * st];
}
__device__ __forceinline__ void put_line(double* o, int st, const double d[7]) {
#pragma unroll
    for (int q = 0; q < 7; q++) o[q * st] = d[q];
}

// The variables of a pass: which array and which scratch pair each starts at,
// those with second derivatives first.
struct CubeVars {
    uint8_t var[NVARS], pair[NVARS];
    int n2, n;
};
inline CubeVars cube_vars(const ColVars& v) {
    CubeVars c = {};
    auto add = [&](int step) {
        c.var[c.n] = (uint8_t)stage_order(step);
        c.pair[c.n++] = (uint8_t)pair_base(step);
    };
    for (int i = 0; i < v.n2; i++) add(v.second[i]);
    c.n2 = c.n;
    for (int i = 0; i < v.n1; i++) add(v.first[i]);
    return c;
}

// One variable of one block.  w: its first scratch pair of the block's zones,
// pairs zs apart; ex: extents of the zones to write.  The three groups run the
// same code on lines along x, y and z.
template <bool ZIP>
__device__ __forceinline__ void cube_variable(const double* __restrict__ src, const BssnBlockDesc& blk,
                                              const int ex[3], bool second, const AxisCoef* cfs,
                                              double2* __restrict__ w, int64_t zs, const ZipGrid& g, double* sm) {
    constexpr int S = Cube::S, UP = Cube::UP, XP = Cube::XP, HP = Cube::HP;
    double* dx = sm + Cube::U;
    double* dy = dx + Cube::DX;
    double *z0 = dy + Cube::DY, *z1 = z0 + Cube::Z, *z2 = z1 + Cube::Z;  // single values of the zones
    const int tid = threadIdx.x, h = tid >> 6;
    // the line's place across the two other axes: a along the lower one
    const int a = tid & 7, b = tid >> 3 & 7;
    const bool line = a < 7 && b < 7;
    {
        // point tid of every plane; without second derivatives only the block's
        // own columns of the halo planes
        const int y = div_small(tid, 1.0f / S), x = tid - S * y;
        bool on = tid < S * S, halo = on && (second || (x >= PW && x < PW + 7 && y >= PW && y < PW + 7));
        const double* p = src + tid;
        const int64_t zst = ZIP ? (int64_t)g.gx * g.gy : S * S;
        bool in = true;
        int zg = 0;
        if (ZIP) {
            const int X = blk.g0[0] + x - PW, Y = blk.g0[1] + y - PW;
            in = X >= 0 && Y >= 0 && X < g.gx && Y < g.gy;
            zg = blk.g0[2] - PW;
            p = src + (in ? X + (int64_t)g.gx * Y : 0) + zst * zg;
        }
#pragma unroll
        for (int z = 0; z < S; z++) {
            if (z < PW || z >= PW + 7 ? halo : on) {
                if (!ZIP || (in && zg + z >= 0 && zg + z < g.gz))
                    cp_async8(sm + z * UP + tid, ZIP ? p + zst * z : p + z * S * S);
                else
                    sm[z * UP + tid] = 0.0;
            }
        }
    }
    cp_async_commit();
    col_wait_pending<0>();
    __syncthreads();
    const unsigned face = blk.bflag >> (2 * h) & 3u;
    double d1[7], d2[7], ko[7];
    if (line) {
        double r[13];
        get_line(r, sm + (h == 2 ? (b + PW) * S + a + PW : (b + PW) * UP + (h ? a + PW : (a + PW) * S)),
                 h == 0 ? 1 : h == 1 ? S : UP);
        line_all(r, face, second, cfs[h], d1, d2, ko);
        const int zx = b * HP + a * 7, zy = b * HP + a, zz = b * 7 + a;  // place of zone q: + 1, 7, HP a step
        if (h == 0) {
            put_line(dx + (b + PW) * XP + (a + PW) * 7, 1, d1);
        }
        if (h == 0) put_line(z0 + zx, 1, ko);
        if (h == 0 && second) put_line(z2 + zx, 1, d2);
        if (h == 1 && second) put_line(dy + (b + PW) * HP + a, 7, d1);
        if (h == 1 && !second) put_line(z1 + zy, 7, ko);
        if (h == 2 && second) {
            put_line(z1 + zz, HP, ko);
            if (a < ex[0] && b < ex[1])
#pragma unroll
                for (int q = 0; q < 7; q++)
                    if (q < ex[2]) w[2 * zs + a + 7 * b + 49 * q] = make_double2(d1[q], d2[q]);
        }
    }
    if (second) {
        // first derivatives on the halo rows that the mixed ones read: d/dx on
        // rows y of the block's planes (a: 0..5, b: plane) and on the halo planes
        // (a: row, b: 0..5), d/dy on the halo planes
        const int ah = a < PW ? a : a + 7, bh = b < PW ? b : b + 7;
        if (h == 0 ? a < 6 && b < 7 : a < 7 && b < 6) {
            double r[13], d[7];
            const int row = h == 0 ? ah : a + PW, plane = h == 0 ? b + PW : bh;
            get_line(r, sm + plane * UP + (h == 2 ? row : row * S), h == 2 ? S : 1);
            const int ax = h == 2 ? 1 : 0;
            line_d1<false>(r, blk.bflag >> (2 * ax) & 3u, cfs[ax], d);
            put_line(h == 2 ? dy + plane * HP + a : dx + plane * XP + row * 7, h == 2 ? 7 : 1, d);
        }
    }
    __syncthreads();
    if (second) {
        double r[13], m[7];
        if (line) {
            // d/dx along y (xy), d/dx along z (xz), d/dy along z (yz)
            get_line(r, h == 1 ? dx + (b + PW) * XP + a : h == 2 ? dx + (b + PW) * 7 + a : dy + b * 7 + a,
                     h == 1 ? 7 : h == 2 ? XP : HP);
            const int ax = h == 1 ? 1 : 2;
            line_d1<true>(r, blk.bflag >> (2 * ax) & 3u, cfs[ax], m);
            const int zy = b * HP + a, zz = b * 7 + a;
            if (h == 0) {
                put_line(sm + zz, HP, m);  // the cube has been read
                if (a < ex[0] && b < ex[1])
#pragma unroll
                    for (int q = 0; q < 7; q++)
                        if (q < ex[2])
                            w[a + 7 * b + 49 * q] = make_double2(dx[(q + PW) * XP + (b + PW) * 7 + a], r[PW + q]);
            }
            if (h == 1 && a < ex[0] && b < ex[2])
#pragma unroll
                for (int q = 0; q < 7; q++)
                    if (q < ex[1]) {
                        double2* o = w + a + 49 * b + 7 * q;
                        o[zs] = make_double2(z2[zy + 7 * q], d2[q]);
                        o[4 * zs] = make_double2(m[q], z0[zy + 7 * q] + ko[q] + z1[zy + 7 * q]);
                    }
        }
        __syncthreads();
        if (line && h == 2 && a < ex[0] && b < ex[1])
#pragma unroll
            for (int q = 0; q < 7; q++)
                if (q < ex[2])
                    w[3 * zs + a + 7 * b + 49 * q] = make_double2(m[q], sm[b * 7 + a + HP * q]);
    } else if (line) {
        if (h == 1 && a < ex[0] && b < ex[2])
#pragma unroll
            for (int q = 0; q < 7; q++)
                if (q < ex[1])
                    w[a + 49 * b + 7 * q] = make_double2(dx[(b + PW) * XP + (q + PW) * 7 + a], d1[q]);
        if (h == 2 && a < ex[0] && b < ex[1])
#pragma unroll
            for (int q = 0; q < 7; q++)
                if (q < ex[2])
                    w[zs + a + 7 * b + 49 * q] =
                        make_double2(d1[q], z0[b * 7 + a + HP * q] + z1[b * 7 + a + HP * q] + ko[q]);
    }
}

template <bool ZIP>
__device__ __forceinline__ void cube_cta(const ConstVars& u, const BrickTask& tk, const BssnBlockDesc& blk,
                                         const AxisCoef* axis, int task, int v, double* __restrict__ S, int64_t zs,
                                         const ZipGrid& g, const CubeVars& vars) {
    extern __shared__ __align__(16) double smem[];
    __shared__ AxisCoef cfs[3];
    const int tid = threadIdx.x;
    if (tid < 24) (&cfs[0].ih60)[tid] = (&axis[0].ih60)[tid];
    int ex[3];
    owned_extent(blk, tk, g, false, ex);
    cube_variable<ZIP>(u.p[vars.var[v]] + (ZIP ? 0 : blk.offset), blk, ex, v < vars.n2, cfs,
                       reinterpret_cast<double2*>(S) + (int64_t)task * Cube::ZONES + (int64_t)vars.pair[v] * zs, zs, g,
                       smem);
}

// The lists' n blocks times the pass's variables.
template <bool ZIP>
__global__ void __launch_bounds__(Cube::T, 4)
cube_kernel(const __grid_constant__ ConstVars u, const BssnBlockDesc* __restrict__ blocks,
            const AxisCoef* __restrict__ axis, const BrickTask* __restrict__ tasks, int n, double* __restrict__ S,
            int64_t zs, ZipGrid g, const __grid_constant__ CubeVars vars) {
    const int per = kCubeGroup * vars.n, first = blockIdx.x / per * kCubeGroup;
    const int q = blockIdx.x % per, m = min(kCubeGroup, n - first);
    const int v = q / m, task = first + q % m;
    const BrickTask tk = tasks[task];
    cube_cta<ZIP>(u, tk, blocks[tk.blk], axis + 3 * (int64_t)tk.blk, task, v, S, zs, g, vars);
}

// One block.
__global__ void __launch_bounds__(Cube::T, 4)
cube_one_kernel(const __grid_constant__ ConstVars u, const __grid_constant__ SplitOne one, double* __restrict__ S,
                int64_t zs, const __grid_constant__ CubeVars vars) {
    cube_cta<false>(u, one_brick(Cube::S, 0, Cube::N, Cube::N), one.blk, one.axis, 0, blockIdx.x, S, zs,
                    ZipGrid{0, 0, 0}, vars);
}

// Host replay of cube_variable's shared-memory indexing: places outside their
// array, counted.
long cube_selfcheck() {
    constexpr int S = Cube::S, UP = Cube::UP, XP = Cube::XP, HP = Cube::HP;
    long bad = 0;
    auto line = [&](int first, int st, int n, int size) {
        if (first < 0 || first + (n - 1) * st >= size) bad++;
    };
    for (int tid = 0; tid < Cube::T; tid++) {
        const int h = tid >> 6, a = tid & 7, b = tid >> 3 & 7;
        const int ah = a < PW ? a : a + 7, bh = b < PW ? b : b + 7;
        if (tid < S * S) line(tid, UP, S, Cube::U);
        if (a < 7 && b < 7) {
            line(h == 2 ? (b + PW) * S + a + PW : (b + PW) * UP + (h ? a + PW : (a + PW) * S),
                 h == 0 ? 1 : h == 1 ? S : UP, 13, Cube::U);
            line((b + PW) * XP + (a + PW) * 7, 1, 7, Cube::DX);
            line((b + PW) * HP + a, 7, 7, Cube::DY);
            line(b * HP + a * 7, 1, 7, Cube::Z);
            line(b * HP + a, 7, 7, Cube::Z);
            line(b * 7 + a, HP, 7, Cube::Z);
            line(h == 1 ? (b + PW) * XP + a : (b + PW) * 7 + a, h == 1 ? 7 : XP, 13, Cube::DX);
            line(b * 7 + a, HP, 13, Cube::DY);
        }
        if (h == 0 ? a < 6 && b < 7 : a < 7 && b < 6) {
            const int row = h == 0 ? ah : a + PW, plane = h == 0 ? b + PW : bh;
            line(plane * UP + (h == 2 ? row : row * S), h == 2 ? S : 1, 13, Cube::U);
            if (h == 2)
                line(plane * HP + a, 7, 7, Cube::DY);
            else
                line(plane * XP + row * 7, 1, 7, Cube::DX);
        }
    }
    return bad;
}

}  // namespace
}  // namespace bssn
