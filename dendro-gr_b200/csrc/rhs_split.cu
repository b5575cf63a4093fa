// Split BSSN right-hand side: a derivative pass, then a pointwise equation
// pass, over brick task lists.
//
// The fused kernel keeps every derivative of a zone in registers; its code is
// one straight run of all 24 variables (about 1 MB of instructions) at 255
// registers and one CTA per SM, so it stalls on instruction fetch and on
// FP64 latency.  Here:
//   * column_kernel (rhs_columns.cuh) marches columns of each variable along
//     z, or cube_kernel (rhs_cube.cuh) takes whole 13^3 blocks, and writes every zone's gradient, second derivatives and summed KO
//     term to a scratch array;
//   * eq_kernel evaluates the equations per zone (rhs_equations.cuh, the same
//     code as the fused kernel) reading those derivatives back.
// The scratch holds slot pairs, [pair][task * NZ + zone][2], so both passes
// move 16-byte pairs in whole rows of consecutive zones.  A task list longer
// than the scratch is processed in chunks, each a derivative launch followed
// by an equation launch on the same stream.
//
// Derivatives are bit-identical to the fused kernel's (same stencils); the
// equations are the same code, so both paths give the same RHS.
#include <cuda_runtime.h>

#include <algorithm>

#include "bssn_common.cuh"
#include "pool.h"
#include "rhs_brick.cuh"
#include "rhs_columns.cuh"
#include "rhs_cube.cuh"
#include "rhs_equations.cuh"
#include "rhs_fused.cuh"

namespace bssn {

namespace {

// equation pass: variables whose derivatives are in flight ahead of use, and
// the per-thread ring of scratch pairs (shared memory) they land in; one
// variable more than the prefetch distance, so a copy never targets a row
// read by the variable just consumed
constexpr int kPrefetchSteps = 6;
constexpr int kRingPairs = (kPrefetchSteps + 1) * kPairsSecond;
constexpr int kEqThreads = 128;

template <int N>
__device__ __forceinline__ void cp_async_wait_pending() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

// One thread per zone, kEqThreads zones of a brick per CTA (a brick of NZ
// zones takes ceil(NZ / kEqThreads) CTAs), so two CTAs share an SM at 254
// registers.  Each thread streams its own zone's 24 variables and scratch
// slots into its own columns of shared memory with cp.async, the slots
// kPrefetchSteps variables ahead of the equations that consume them (one
// commit group per variable; a thread only reads what it copied itself, so
// no barrier).
// g.gx == 0: variables and right-hand sides at the zone's padded index.
// g.gx > 0: only zones owning their node run and write the right-hand side
// at the node index of the zipped grid; the variables are read there too
// (zip_in, direct form) or at the padded index.
// bx, by, nz: rows and zones of a brick in the scratch; part: the CTA's
// kEqThreads zones of the brick.
__device__ __forceinline__ void eq_cta(const RhsArgs& A, const BrickTask& tk, const BssnBlockDesc& blk, int task,
                                       int part, const double* __restrict__ S, int64_t zs, const ZipGrid& g,
                                       int zip_in, int bx, int by, int nz) {
    extern __shared__ __align__(16) double ring[];  // [kRingPairs][T][2] | vals [NVARS][T]
    const int tid = threadIdx.x;
    const int o[3] = {tk.o[0], tk.o[1], tk.o[2]};
    // the zones that run: the brick's extent, or on the zipped grid only the
    // zones owning their node; the threads are packed onto them, so no lane
    // idles on a skipped zone
    int ex[3];
    owned_extent(blk, tk, g, false, ex);
    const int j = part * kEqThreads + tid;  // the thread's zone among them
    if (j >= ex[0] * ex[1] * ex[2]) return;
    const int r0 = j % ex[0], r1 = (j / ex[0]) % ex[1], r2 = j / (ex[0] * ex[1]);
    const int l = r0 + bx * (r1 + by * r2);  // zone index in the brick (scratch position)
    const int za0 = o[0] + PW + r0, za1 = o[1] + PW + r1, za2 = o[2] + PW + r2;
    const int64_t pidx = blk.offset + za0 + (int64_t)blk.sz * (za1 + (int64_t)blk.sz * za2);
    int64_t node = pidx;
    if (g.gx)
        node = (blk.g0[0] + za0 - PW) +
               (int64_t)g.gx * ((blk.g0[1] + za1 - PW) + (int64_t)g.gy * (blk.g0[2] + za2 - PW));
    const int64_t in_idx = zip_in ? node : pidx;
    const double2* in = reinterpret_cast<const double2*>(S) + (int64_t)task * nz + l;
    double2* col = reinterpret_cast<double2*>(ring) + tid;   // this thread's ring column
    double* vals = ring + 2 * kRingPairs * kEqThreads + tid;  // [NVARS][kEqThreads]
    // the zone's 24 variables first, as their own commit group
#pragma unroll
    for (int v = 0; v < NVARS; v++) cp_async8(vals + v * kEqThreads, A.u.p[v] + in_idx);
    cp_async_commit();
    // pair P of the zone lives in ring row P % kRingPairs
    auto issue = [&](int step) {
        if (step < NVARS) {
            const int b = pair_base(step), n = stage_second(step) ? kPairsSecond : kPairsFirst;
#pragma unroll
            for (int q = 0; q < kPairsSecond; q++)
                if (q < n) cp_async16(col + ((b + q) % kRingPairs) * kEqThreads, in + (int64_t)(b + q) * zs);
        }
        cp_async_commit();  // empty groups past the last variable keep the count fixed
    };
#pragma unroll
    for (int k = 0; k < kPrefetchSteps; k++) issue(k);
    cp_async_wait_pending<kPrefetchSteps>();  // the variables' group
    auto pv = [&](int v) { return vals[v * kEqThreads]; };
    int step = 0;
    auto get = [&](auto tag, double* d1, double* d2, double& ko) {
        constexpr bool SECOND = decltype(tag)::value;
        cp_async_wait_pending<kPrefetchSteps - 1>();
        const int b = pair_base(step);
        auto rd = [&](int q) { return col[((b + q) % kRingPairs) * kEqThreads]; };
        const double2 p0 = rd(0);  // dx dy
        d1[0] = p0.x;
        d1[1] = p0.y;
        if (SECOND) {
            const double2 p1 = rd(1), p2 = rd(2), p3 = rd(3), p4 = rd(4);  // xx yy | dz zz | xz yz | xy ko
            d1[2] = p2.x;
            d2[0] = p1.x;
            d2[1] = p4.x;
            d2[2] = p3.x;
            d2[3] = p1.y;
            d2[4] = p3.y;
            d2[5] = p2.y;
            ko = p4.y;
        } else {
            const double2 p1 = rd(1);  // dz ko
            d1[2] = p1.x;
            ko = p1.y;
        }
        issue(step + kPrefetchSteps);  // rows of variables consumed before this one
        step++;
    };
    auto store = [&](int v, double r) { A.rhs.p[v][node] = r; };
    zone_equations(A, blk, za0, za1, za2, get, pv, store);
}

__global__ void __launch_bounds__(kEqThreads, 2)
eq_kernel(RhsArgs A, const BssnBlockDesc* __restrict__ blocks,
          const BrickTask* __restrict__ tasks, const double* __restrict__ S, int64_t zs,
          ZipGrid g, int zip_in, int bx, int by, int nz) {
    const int parts = (nz + kEqThreads - 1) / kEqThreads, task = blockIdx.x / parts;
    const BrickTask tk = tasks[task];
    const BssnBlockDesc blk = blocks[tk.blk];
    eq_cta(A, tk, blk, task, blockIdx.x % parts, S, zs, g, zip_in, bx, by, nz);
}

// The bricks of one block.
__global__ void __launch_bounds__(kEqThreads, 2)
eq_one_kernel(RhsArgs A, const __grid_constant__ SplitOne one, const double* __restrict__ S, int64_t zs, int bx,
              int by, int nz) {
    const int parts = (nz + kEqThreads - 1) / kEqThreads, task = blockIdx.x / parts;
    const BrickTask tk = one_brick(one.blk.sz, task, bx, by);
    eq_cta(A, tk, one.blk, task, blockIdx.x % parts, S, zs, ZipGrid{0, 0, 0}, 0, bx, by, nz);
}

constexpr size_t eq_smem_bytes() { return sizeof(double) * kEqThreads * (2 * kRingPairs + NVARS); }

struct SplitEntry {
    int bx, by, v2, g2, v1, g1, threads, iter, hit, plane, dx_plane;
    size_t smem;
    void (*deriv_one)(ConstVars, SplitOne, double*, int64_t, int, ColVars);
    void (*deriv)(ConstVars, const BssnBlockDesc*, const AxisCoef*, const BrickTask*, double*, int64_t, ZipGrid, int,
                  ColVars);
    void (*deriv_zip)(ConstVars, const BssnBlockDesc*, const AxisCoef*, const BrickTask*, double*, int64_t, ZipGrid, int,
                  ColVars);
};

template <int BX, int BY>
SplitEntry make_split() {
    using Sh = ColShape<BX, BY>;
    return SplitEntry{BX, BY, Sh::V2, Sh::G2, Sh::V1, Sh::G1, Sh::T, Sh::ITER, Sh::HIT, Sh::PL, Sh::DXP,
                      Sh::SMEM, column_one_kernel<Sh>, column_kernel<Sh, false>, column_kernel<Sh, true>};
}

// brick shapes (columns; every brick has its block's whole height), in the
// order of the tile table's split tiles (rhs_fused.cu)
const SplitEntry* split_table(int* count) {
    static const SplitEntry table[] = {
        make_split<8, 8>(),  make_split<7, 7>(),   make_split<8, 4>(),   make_split<13, 5>(),
        make_split<9, 9>(),  make_split<13, 13>(), make_split<25, 9>(), make_split<49, 10>(),
    };
    *count = (int)(sizeof(table) / sizeof(table[0]));
    return table;
}

// Whole 13^3 blocks run the cube form of the derivative pass, padded or from
// the node grid, few or many, with faces or without (64 blocks 14 us, 25 as
// columns; 8,000 blocks 1.57 ms, 1.97).
bool takes_cube(const SplitEntry& t, int side) { return side == Cube::S && t.bx == Cube::N && t.by == Cube::N; }

}  // namespace

int split_shape_count() {
    int c;
    split_table(&c);
    return c;
}

int split_columns(int shape, int b[2]) {
    int c;
    const SplitEntry* t = split_table(&c);
    if (shape < 0 || shape >= c) return BSSN_EINVAL;
    b[0] = t[shape].bx;
    b[1] = t[shape].by;
    return 0;
}

int split_threads(int shape) {
    int c;
    const SplitEntry* t = split_table(&c);
    return (shape < 0 || shape >= c) ? 0 : t[shape].threads;
}

size_t split_smem(int shape) {
    int c;
    const SplitEntry* t = split_table(&c);
    return (shape < 0 || shape >= c) ? 0 : t[shape].smem;
}

// Host replay of column_march's shared-memory indexing: every brick the
// splitter makes of every block side the shape takes, with and without the
// layers another block owns, with every face of the block physical or none.
// Returns the number of variable groups that do not fit the CTA's threads and
// buffers, of taps outside the staged planes and of places outside the ring
// slots, the d/dx planes or the brick's scratch.
long split_selfcheck(int shape) {
    int c;
    const SplitEntry* tab = split_table(&c);
    if (shape < 0 || shape >= c) return -1;
    const SplitEntry& t = tab[shape];
    const int B[2] = {t.bx, t.by}, TX = t.bx + 2 * PW, T = t.threads;
    long bad = 0;
    if (t.v2 * t.g2 < kSecondVars || t.v1 * t.g1 < kFirstVars) bad++;
    if (takes_cube(t, Cube::S)) bad += cube_selfcheck();
    auto case_of = [](int a, int s, int faces) {  // -1: centred
        if (!faces) return -1;
        return a <= 5 ? a - 3 : a >= s - 6 ? a - (s - 9) : -1;
    };
    for (int s : {13, 19, 31, 55})
        for (int own = 0; own < 2; own++)
            for (int faces = 0; faces < 2; faces++) {
                const int n = s - 2 * PW;
                const int nb[2] = {(n + B[0] - 1) / B[0], (n + B[1] - 1) / B[1]};
                for (int q = 0; q < nb[0] * nb[1]; q++) {
                    int o[2], e[2];
                    const int qq[2] = {q % nb[0], q / nb[0]};
                    for (int d = 0; d < 2; d++) {
                        split1(n, B[d], qq[d], o[d], e[d]);
                        if (e[d] < 3) bad++;  // a closure reads five points inward
                        if (own && !faces && o[d] + e[d] == n) e[d]--;
                        if (e[d] < 1 || e[d] > B[d]) bad++;
                    }
                    const int sx = e[0] + 2 * PW, sy = e[1] + 2 * PW, cols = e[0] * e[1];
                    for (int kind = 0; kind < 2; kind++) {
                        const int nv = kind ? t.v1 : t.v2;
                        const int ring = kColRing * nv * t.plane;
                        const int rings = kind ? ring : ring + kColRing * nv * (t.dx_plane + t.bx * t.by);
                        if (nv * cols > T || nv * sx * sy > t.iter * T) bad++;
                        if (!kind && nv * 2 * PW * e[0] > t.hit * T) bad++;
                        if (rings > (int)(t.smem / sizeof(double))) bad++;
                    }
                    // taps of a column along x and y stay in the staged plane
                    for (int d = 0; d < 2; d++)
                        for (int i = 0; i < e[d]; i++) {
                            const int a = o[d] + PW + i, cs = case_of(a, s, faces);
                            const int lo = cs < 0 ? i : (cs < 3 ? 3 : s - 9) - o[d];
                            const int hi = cs < 0 ? i + 2 * PW : lo + 5;
                            if (lo < 0 || hi >= e[d] + 2 * PW) bad++;
                        }
                    if ((sy - 1) * TX + sx - 1 >= t.plane) bad++;
                    if ((sy - 1) * t.bx + e[0] - 1 >= t.dx_plane) bad++;
                    if (e[0] - 1 + t.bx * (e[1] - 1 + t.by * (n - 1)) >= t.bx * t.by * n) bad++;
                }
            }
    return bad;
}

int prepare_split(int shape) {
    int c;
    const SplitEntry* t = split_table(&c);
    if (shape < 0 || shape >= c) return BSSN_EINVAL;
    int st = set_smem_limit((const void*)t[shape].deriv, (int)t[shape].smem);
    if (!st) st = set_smem_limit((const void*)t[shape].deriv_one, (int)t[shape].smem);
    if (!st) st = set_smem_limit((const void*)t[shape].deriv_zip, (int)t[shape].smem);
    if (!st && takes_cube(t[shape], Cube::S)) {
        st = set_smem_limit((const void*)cube_kernel<false>, (int)Cube::SMEM);
        if (!st) st = set_smem_limit((const void*)cube_kernel<true>, (int)Cube::SMEM);
        if (!st) st = set_smem_limit((const void*)cube_one_kernel, (int)Cube::SMEM);
    }
    if (!st) st = set_smem_limit((const void*)eq_kernel, (int)eq_smem_bytes());
    if (!st) st = set_smem_limit((const void*)eq_one_kernel, (int)eq_smem_bytes());
    return st;
}

int split_shape_chunks(int shape, int side, const ConstVars& u, const AxisCoef* axis,
                       const BssnBlockDesc* blocks_dev, const BrickTask* tasks_dev, int ntasks, double* scratch,
                       int64_t scratch_zones, cudaStream_t s, const ZipGrid& g, const ColVars& vars, bool zip_in,
                       KernelTimer* tm, const ChunkWork& after) {
    int c;
    const SplitEntry* tab = split_table(&c);
    if (shape < 0 || shape >= c || side <= 2 * PW || !axis) return BSSN_EINVAL;
    if (ntasks <= 0) return 0;
    const SplitEntry& t = tab[shape];
    const int b[2] = {t.bx, t.by};
    const int nz = t.bx * t.by * (side - 2 * PW);  // zones of a brick in the scratch
    const int64_t chunk = scratch ? scratch_zones / nz : 0;
    if (chunk <= 0) return BSSN_EINVAL;
    int st = prepare_split(shape);
    if (st) return st;
    const int groups = col_groups(vars.n2, t.v2) + col_groups(vars.n1, t.v1);
    const int64_t zs = chunk * nz;  // slot stride
    for (int64_t c0 = 0; c0 < ntasks; c0 += chunk) {
        const int n = (int)(ntasks - c0 < chunk ? ntasks - c0 : chunk);
        if (tm && (st = tm->start(KernelTimer::DERIV, s))) return st;
        if (takes_cube(t, side))
            (zip_in ? cube_kernel<true> : cube_kernel<false>)<<<n * (vars.n2 + vars.n1), Cube::T, Cube::SMEM, s>>>(
                u, blocks_dev, axis, tasks_dev + c0, n, scratch, zs, g, cube_vars(vars));
        else
            (zip_in ? t.deriv_zip : t.deriv)<<<n * groups, t.threads, t.smem, s>>>(
                u, blocks_dev, axis, tasks_dev + c0, scratch, zs, g, nz, vars);
        st = cuda_status(cudaGetLastError());
        if (!st && tm) st = tm->stop(s);
        if (!st) st = after(tasks_dev + c0, n, zs, b, nz);
        if (st) return st;
    }
    return 0;
}

static ColVars all_vars() {
    ColVars all = {};
    for (int i = 0; i < kSecondVars; i++) all.second[all.n2++] = (uint8_t)second_step(i);
    for (int i = 0; i < kFirstVars; i++) all.first[all.n1++] = (uint8_t)first_step(i);
    return all;
}

// One block through the two passes: the same kernels, hence the same bits, as
// a mesh's block.  The fused kernel that served these calls runs a megabyte of
// straight-line code once and waits for its instructions: 184 us for a 13^3
// block and 482 for a 55^3 one, here 41 and 117.  BSSN_ENOMEM before any
// launch when the scratch cannot be had (a stream capture, which would record
// the allocation, or no memory): the caller then runs the fused kernel.
int launch_rhs_split_single(int shape, const RhsArgs& A, const BssnBlockDesc& blk, cudaStream_t s) {
    int c;
    const SplitEntry* tab = split_table(&c);
    if (shape < 0 || shape >= c) return BSSN_EINVAL;
    const SplitEntry& t = tab[shape];
    int st = prepare_split(shape);
    if (st) return st;
    const int n = blk.sz - 2 * PW;
    const int bricks = ((n + t.bx - 1) / t.bx) * ((n + t.by - 1) / t.by);
    const int nz = t.bx * t.by * n;
    const int64_t zs = (int64_t)bricks * nz;
    double* scratch = nullptr;
    st = pool_alloc((void**)&scratch, sizeof(double) * kSplitSlots * zs, s);
    if (st) return st;
    SplitOne one;
    one.blk = blk;
    for (int d = 0; d < 3; d++) one.axis[d] = axis_coef((blk.ptmax[d] - blk.ptmin[d]) / (blk.sz - 1));
    const ColVars all = all_vars();
    if (takes_cube(t, blk.sz))
        cube_one_kernel<<<all.n2 + all.n1, Cube::T, Cube::SMEM, s>>>(A.u, one, scratch, zs, cube_vars(all));
    else
        t.deriv_one<<<bricks * (t.g2 + t.g1), t.threads, t.smem, s>>>(A.u, one, scratch, zs, nz, all);
    st = cuda_status(cudaGetLastError());
    if (!st) {
        const int parts = (nz + kEqThreads - 1) / kEqThreads;
        eq_one_kernel<<<bricks * parts, kEqThreads, eq_smem_bytes(), s>>>(A, one, scratch, zs, t.bx, t.by, nz);
        st = cuda_status(cudaGetLastError());
    }
    const int fr = pool_free(scratch, s);
    return st ? st : fr;
}

int launch_rhs_split(int shape, const RhsArgs& A, const BssnBlockDesc* blocks_dev,
                     const BrickTask* tasks_dev, int ntasks, double* scratch,
                     int64_t scratch_zones, cudaStream_t s, KernelTimer* tm,
                     const int32_t* zip_grid, bool zip_in, int side) {
    const ZipGrid g = zip_grid ? ZipGrid{zip_grid[0], zip_grid[1], zip_grid[2]} : ZipGrid{0, 0, 0, A.drop};
    zip_in = zip_in && zip_grid;
    const ColVars all = all_vars();
    return split_shape_chunks(
        shape, side, A.u, A.axis, blocks_dev, tasks_dev, ntasks, scratch, scratch_zones, s, g, all, zip_in, tm,
        [&](const BrickTask* tasks, int n, int64_t zs, const int b[2], int nz) {
            int st = 0;
            if (tm && (st = tm->start(KernelTimer::EQ, s))) return st;
            const int parts = (nz + kEqThreads - 1) / kEqThreads;
            eq_kernel<<<n * parts, kEqThreads, eq_smem_bytes(), s>>>(A, blocks_dev, tasks, scratch, zs, g,
                                                                     zip_in ? 1 : 0, b[0], b[1], nz);
            st = cuda_status(cudaGetLastError());
            if (!st && tm) st = tm->stop(s);
            return st;
        });
}

}  // namespace bssn
