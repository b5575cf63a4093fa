"""The split right-hand side's derivative pass (columns marched along z) where
its indexing can go wrong: every block side, with no face, single faces,
edges and all six faces physical, under every split tile, against the oracle
on noise around the flat metric; padding beyond physical faces, which the
reference never reads, holds NaN."""
import ctypes as C

import numpy as np
import pytest

import oracle_lib as ol

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

FLAGS = (0, 1, 2, 4, 8, 16, 32, 21, 42, 63)


def _blocks(B, side):
    """One block per face set, next to each other in memory only."""
    blocks = (B.BssnBlockDesc * len(FLAGS))()
    h = 1.0 / 6.0
    for b, fl in enumerate(FLAGS):
        blk = blocks[b]
        blk.offset, blk.sz, blk.bflag = b * ((side ** 3 + 1) // 2 * 2), side, fl
        for k in range(3):
            blk.g0[k] = 0
            blk.ptmin[k] = 0.3 * (b - 4) + 0.1 * k - 3 * h
            blk.ptmax[k] = blk.ptmin[k] + (side - 1) * h
    G = (6 * ((side - 7) // 6) + 1,) * 3
    return B.MeshSpec(blocks, len(FLAGS), G, h, 0.0, np.full(len(FLAGS), side, dtype=np.int32))


@pytest.mark.parametrize("side", [13, 19, 31, 55])
def test_every_face_set_and_split_tile(side):
    import bssn_b200 as B
    spec = _blocks(B, side)
    rng = np.random.default_rng(side)
    U = np.zeros((24, spec.n_unzip))
    U[[0, 1, 12, 15, 17]] = 1.0
    U += 1e-3 * rng.uniform(-1, 1, U.shape)
    ref = np.zeros_like(U)
    for b in range(spec.nblocks):
        blk = spec.blocks[b]
        n = side ** 3
        v = np.ascontiguousarray(U[:, int(blk.offset):int(blk.offset) + n])
        r = ol.oracle().bssnrhs(v, 0, np.array(list(blk.ptmin)), np.array(list(blk.ptmax)), side, int(blk.bflag),
                                ol.params())
        ref[:, int(blk.offset):int(blk.offset) + n] = np.asarray(r).reshape(24, n)
        cube = v.reshape(24, side, side, side)
        for axis in range(3):  # x is the last axis
            ax = 3 - axis
            if blk.bflag >> (2 * axis) & 1:
                cube[(slice(None),) * ax + (slice(0, 3),)] = np.nan
            if blk.bflag >> (2 * axis + 1) & 1:
                cube[(slice(None),) * ax + (slice(side - 3, side),)] = np.nan
        U[:, int(blk.offset):int(blk.offset) + n] = v
    mask = np.zeros(spec.n_unzip, dtype=bool)
    for b in range(spec.nblocks):
        m = np.zeros((side,) * 3, dtype=bool)
        m[3:-3, 3:-3, 3:-3] = True
        off = int(spec.blocks[b].offset)
        mask[off:off + side ** 3] = m.reshape(-1)
    mesh = B.Mesh(spec)
    dU = torch.from_numpy(U).cuda()
    split = [t for t in range(len(B.tiles())) if B.tile_mode(t) == 1]
    first = None
    for t in [-1] + split:
        dR = torch.zeros_like(dU)
        mesh.rhs(dR, dU, B.default_params(), tile=t)
        torch.cuda.synchronize()
        got = dR.cpu().numpy()[:, mask]
        # the bound of every right-hand-side test: 1e-12 of the variable's largest value
        err = ol.rel_err(ref[:, mask], got)
        assert err.max() <= 1e-12, (t, err.max(), int(err.argmax()))
        # every tile applies the same stencils and the same equations
        first = got if first is None else first
        assert np.array_equal(first, got), t


@pytest.mark.parametrize("side", [13, 19, 31, 55])
def test_single_block_equals_mesh_block(side):
    """A single-block call runs the mesh's two passes from the library's pool:
    the same bits as the block in a mesh, on two streams at once, and, where a
    stream capture forbids the pool, the one-kernel form's (the same stencils
    and equations: the same bits too)."""
    import bssn_b200 as B
    spec = _blocks(B, side)
    rng = np.random.default_rng(100 + side)
    U = np.zeros((24, spec.n_unzip))
    U[[0, 1, 12, 15, 17]] = 1.0
    U += 1e-3 * rng.uniform(-1, 1, U.shape)
    dU = torch.from_numpy(U).cuda()
    prm = B.default_params()
    mesh = B.Mesh(spec)
    ref = torch.zeros_like(dU)
    mesh.rhs(ref, dU, prm)
    got = torch.zeros_like(dU)
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]

    def call(out, b, stream):
        blk = spec.blocks[b]
        B.bssnrhs_block(out, dU, int(blk.offset), list(blk.ptmin), list(blk.ptmax), side, int(blk.bflag), prm,
                        stream=stream)

    for b in range(spec.nblocks):
        call(got, b, streams[b % 2])
    torch.cuda.synchronize()
    assert torch.equal(got, ref)
    got.zero_()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        call(got, 9, torch.cuda.current_stream())
    g.replay()
    torch.cuda.synchronize()
    o = int(spec.blocks[9].offset)
    assert torch.equal(got[:, o:o + side ** 3], ref[:, o:o + side ** 3])


def test_constraints_with_and_without_scratch():
    """Constraints from the derivative scratch and, captured on a mesh that has
    none yet, from the padded block directly: the outer stage of the mixed
    derivatives is rounded differently, 1e-12 of the largest value."""
    import bssn_b200 as B
    spec = B.generate_mesh(1, (1, 1, 1), seed=8, xmin=-8.25)
    U = torch.zeros((24, spec.n_nodes), dtype=torch.float64, device="cuda")
    B.initial_data(U, spec, eps=1e-6)
    out = []
    for captured in (True, False):
        mesh = B.Mesh(spec)
        P = torch.zeros((24, mesh.n_unzip), dtype=torch.float64, device="cuda")
        mesh.unzip(P, U)
        cons = torch.zeros((4, spec.n_nodes), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        if captured:
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g):
                B.constraints(mesh, cons, P)
            g.replay()
        else:
            B.constraints(mesh, cons, P)
        torch.cuda.synchronize()
        out.append(cons.cpu().numpy())
    assert ol.rel_err(out[0], out[1]).max() <= 1e-12


def test_cube_form_over_more_blocks_than_a_group():
    """13^3 blocks in a list longer than the cube form's group of blocks, the
    last group a part of one, on boundary, edge, corner and interior blocks:
    the same bits as columns."""
    import bssn_b200 as B
    spec = B.generate_mesh(0, (11, 11, 11), seed=0, xmin=-8.25)
    U = torch.zeros((24, spec.n_nodes), dtype=torch.float64, device="cuda")
    B.initial_data(U, spec, eps=1e-3)
    mesh = B.Mesh(spec)
    P = torch.zeros((24, mesh.n_unzip), dtype=torch.float64, device="cuda")
    mesh.unzip(P, U)
    cube, cols = torch.zeros_like(P), torch.zeros_like(P)
    mesh.rhs(cube, P, B.default_params(), tile=6)
    mesh.rhs(cols, P, B.default_params(), tile=3)
    torch.cuda.synchronize()
    assert torch.equal(cube, cols)


def _constraints(B, mesh, P, psi4, stream=None):
    n = mesh.spec.n_nodes
    out = torch.zeros((6 if psi4 else 4, n), dtype=torch.float64, device="cuda")
    fn = B.lib.bssn_constraints_psi4_f64 if psi4 else B.lib.bssn_constraints_f64
    fn.argtypes = [C.c_void_p] * 4
    ptrs = (C.c_void_p * out.shape[0])(*[out.data_ptr() + 8 * n * c for c in range(out.shape[0])])
    B.check(fn(mesh.h, B.ptrs(P), ptrs, B.stream_ptr(stream)), "constraints")
    return out


@pytest.mark.parametrize("psi4", [False, True])
def test_captured_constraints_outlive_scratch_growth(psi4):
    """Constraints captured on a mesh that already has derivative scratch,
    replayed after a plan and a right-hand side have replaced that scratch: the
    graph holds nothing of the mesh that can be freed.  The forms with and
    without scratch round the outer stage of the mixed derivatives differently:
    1e-12 of the largest value."""
    import bssn_b200 as B
    spec = B.generate_mesh(1, (2, 2, 2), seed=20261203, xmin=-8.25)
    U = torch.zeros((24, spec.n_nodes), dtype=torch.float64, device="cuda")
    B.initial_data(U, spec, eps=1e-6)
    mesh = B.Mesh(spec)
    P = torch.zeros((24, mesh.n_unzip), dtype=torch.float64, device="cuda")
    mesh.unzip(P, U)
    R = torch.zeros_like(P)
    mesh.rhs(R, P, B.default_params(), tile=6)  # scratch for 7x7 columns
    eager = _constraints(B, mesh, P, psi4)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        captured = _constraints(B, mesh, P, psi4)
    plan = B.RK4Plan(mesh, B.default_params(), B.PLAN_GRAPH)
    mesh.rhs(R, P, B.default_params())
    captured.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert ol.rel_err(eager.cpu().numpy(), captured.cpu().numpy()).max() <= 1e-12
    plan.close()


def test_constraints_over_several_scratch_fuls():
    """1.16 M zones of 13^3 blocks, more than one call's scratch holds, against
    the form without scratch (as above)."""
    import bssn_b200 as B
    spec = B.generate_mesh(0, (15, 15, 15), seed=0, xmin=-8.25)
    assert spec.zones() > 1 << 20
    U = torch.zeros((24, spec.n_nodes), dtype=torch.float64, device="cuda")
    B.initial_data(U, spec, eps=1e-6)
    mesh = B.Mesh(spec)
    P = torch.zeros((24, mesh.n_unzip), dtype=torch.float64, device="cuda")
    mesh.unzip(P, U)
    eager = _constraints(B, mesh, P, True)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        captured = _constraints(B, mesh, P, True)
    g.replay()
    torch.cuda.synchronize()
    assert ol.rel_err(eager.cpu().numpy(), captured.cpu().numpy()).max() <= 1e-12


def test_constraints_beside_right_hand_sides():
    """Constraints on one stream while right-hand sides and steps of the same
    mesh run on another: each has its own scratch, so both give what they give
    alone."""
    import bssn_b200 as B
    spec = B.generate_mesh(1, (2, 1, 1), seed=5, xmin=-8.25)
    U = torch.zeros((24, spec.n_nodes), dtype=torch.float64, device="cuda")
    B.initial_data(U, spec, eps=1e-6)
    prm = B.default_params()
    mesh = B.Mesh(spec)
    P = torch.zeros((24, mesh.n_unzip), dtype=torch.float64, device="cuda")
    mesh.unzip(P, U)
    want_r = torch.zeros_like(P)
    mesh.rhs(want_r, P, prm)
    want_c = _constraints(B, mesh, P, True)
    torch.cuda.synchronize()
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    rhs, cons = [], []
    for _ in range(4):
        rhs.append(torch.zeros_like(P))
        cons.append(torch.zeros_like(want_c))
    torch.cuda.synchronize()
    for k in range(4):
        mesh.rhs(rhs[k], P, prm, stream=a)
        with torch.cuda.stream(b):
            cons[k] = _constraints(B, mesh, P, True, stream=b)
    torch.cuda.synchronize()
    for k in range(4):
        assert torch.equal(rhs[k], want_r) and torch.equal(cons[k], want_c)


def test_captured_right_hand_side_outlives_scratch_growth():
    """A right-hand side captured with the scratch of narrow columns, replayed
    after wider ones and a plan have replaced that scratch, and that plan's own
    graph after another growth."""
    import bssn_b200 as B
    spec = B.generate_mesh(0, (4, 4, 4), seed=0, xmin=-8.25)
    U = torch.zeros((24, spec.n_nodes), dtype=torch.float64, device="cuda")
    B.initial_data(U, spec, eps=1e-6)
    prm = B.default_params()
    mesh = B.Mesh(spec)
    P = torch.zeros((24, mesh.n_unzip), dtype=torch.float64, device="cuda")
    mesh.unzip(P, U)
    want, got = torch.zeros_like(P), torch.zeros_like(P)
    mesh.rhs(want, P, prm, tile=6)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        mesh.rhs(got, P, prm, tile=6)
    for t in range(len(B.tiles())):
        if B.tile_mode(t) == 1:
            mesh.rhs(torch.zeros_like(P), P, prm, tile=t)
    plan = B.RK4Plan(mesh, prm, B.PLAN_GRAPH)
    V = U.clone()
    plan.step(V, 1e-3)
    got.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, want)
    plan.close()


@pytest.mark.parametrize("faces", [True, False])
def test_zipped_steps_under_every_split_tile(faces):
    """A step through the zipped form (node offsets, zero outside the grid,
    owned zones only) under every split tile, on every side that takes it:
    the same bits as the padded block loop, with the domain's physical faces
    and with none (every block interior, zeros beyond the grid)."""
    import bssn_b200 as B
    spec = B.generate_mesh(1, (2, 2, 2), seed=20261203, xmin=-8.25)
    assert set(spec.sides.tolist()) == {13, 19, 31, 55}
    U = torch.zeros((24, spec.n_nodes), dtype=torch.float64, device="cuda")
    B.initial_data(U, spec, eps=1e-6)
    if not faces:
        for b in range(spec.nblocks):
            spec.blocks[b].bflag = 0
    mesh = B.Mesh(spec)
    prm = B.default_params()
    ref = U.clone()
    plan = B.RK4Plan(mesh, prm, B.PLAN_PER_BLOCK)
    plan.step(ref, 1e-6)
    torch.cuda.synchronize()
    plan.close()
    assert bool(torch.isfinite(ref).all()) and not torch.equal(ref, U)
    for flags in (0, B.PLAN_DIRECT):
        plan = B.RK4Plan(mesh, prm, flags)
        for t in range(len(B.tiles())):
            if B.tile_mode(t) != 1:
                continue
            plan.set_tile(t)
            V = U.clone()
            plan.step(V, 1e-6)
            torch.cuda.synchronize()
            assert torch.equal(V, ref), (flags, t)
        plan.close()


def _kernels(f):
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        f()
        torch.cuda.synchronize()
    return {e.name for e in p.events() if "bssn" in e.name}


@pytest.mark.parametrize("flags", [0, 4, 8])  # default, block by block, direct
def test_autotune_times_the_kernels_the_step_runs(flags):
    """Every derivative and equation kernel of a step under the chosen tiles is
    one that the tuner launched to choose them."""
    import bssn_b200 as B
    spec = B.generate_mesh(1, (2, 1, 1), seed=20261203, xmin=-8.25)
    U = torch.zeros((24, spec.n_nodes), dtype=torch.float64, device="cuda")
    B.initial_data(U, spec, eps=1e-6)
    plan = B.RK4Plan(B.Mesh(spec), B.default_params(), flags)
    tuned = _kernels(lambda: plan.autotune(U, reps=1))
    step = {k for k in _kernels(lambda: plan.step(U, 1e-3)) if "column_kernel" in k or "eq_kernel" in k}
    plan.close()
    assert step and step <= tuned, step - tuned


def test_tiles_that_do_not_suit_a_side():
    """Whole-layer tiles of larger blocks leave 13^3 blocks to their default;
    tiles of the same kernel are timed once."""
    import bssn_b200 as B
    spec = B.generate_mesh(0, (2, 2, 2), seed=0, xmin=-8.25)
    U = torch.zeros((24, spec.n_nodes), dtype=torch.float64, device="cuda")
    B.initial_data(U, spec, eps=1e-6)
    plan = B.RK4Plan(B.Mesh(spec), B.default_params())
    for t in (14, 15, 16):
        assert plan.set_tile(t) == {13: 6}
    _, table = plan.autotune(U, reps=1)
    assert table[13][6] == table[13][4] and table[13][7] == table[13][3]
    assert all(table[13][t] > 1e29 for t in (14, 15, 16))
    plan.close()
