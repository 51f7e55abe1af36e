"""The register-resident single-reduction PCG at the edges of its tilings (one
to six rows per thread, grids of a few CTAs) against the global-vector
single-reduction kernel, which performs the same operations row by row with
its vectors in global memory: fields and iteration counts agree bit for bit.
Their grids are the same, so no tolerance is involved."""
import numpy as np
import pytest

from helpers import bitwise, rel_l2

pytestmark = pytest.mark.gpu


def _gpu():
    from cbs3d import gpu
    return gpu


def _same(case, steps=2, **over):
    gpu = _gpu()
    a, b = gpu.Context(case, pcg_kernel=4, **over), gpu.Context(case, pcg_kernel=5, **over)
    sa, sb = a.step(steps), b.step(steps)
    assert sa.pcg_kernel in (4, 9) and sb.pcg_kernel == 8
    assert sa.cg_iterations_total == sb.cg_iterations_total
    assert sa.cg.final_max_abs == sb.cg.final_max_abs and sa.cg.final_l2 == sb.cg.final_l2
    for x, y in zip(a.fields(), b.fields()):
        assert bitwise(x, y)
    a.close()
    b.close()


# 1 slice; a few CTAs; and on 148 SMs the last size of one, two and three rows
# per thread with the first size of the next (41/42, 52/53, 60/61), five (67)
@pytest.mark.parametrize("n", [2, 5, 11, 41, 42, 52, 53, 60, 61, 67])
def test_tilings_match_the_global_vector_kernel(n):
    from cbs3d import cases
    _same(cases.cavity(n, re=400.0, ntime=10 ** 6, jitter=0.15 if n > 2 else 0.0, seed=1234))


@pytest.mark.parametrize("conv_test,abs_tol", [(1, 1e-9), (3, 1e-9)])
def test_stopping_tests_on_the_largest_residual(conv_test, abs_tol):
    """Tests 1 and 3 carry max|r| in every iteration's all-reduce; also against
    the two-reduction kernel, which forms it in its own way."""
    from cbs3d import cases
    gpu = _gpu()
    case = cases.cavity(13, re=100.0, ntime=10 ** 6, cg_conv_test=conv_test, absToler=abs_tol, relToler=1e-9)
    _same(case)
    a, c = gpu.Context(case), gpu.Context(case, pcg_kernel=1)
    sa, sc = a.step(2), c.step(2)
    assert abs(sa.cg.iterations - sc.cg.iterations) <= 2
    # solves to 1e-9 whose sums are grouped differently
    assert rel_l2(a.fields()[1], c.fields()[1]) <= 1e-8


def test_fixed_and_inactive_rows():
    """Outlet rows (fixed pressure) and solid rows (no pressure) stay 0 in the
    recurrences without branches."""
    from cbs3d import cases
    _same(cases.channel(21, 5, 6, ntime=10 ** 6))
    _same(cases.cht_slab(17, 6, 3, 5, ntime=10 ** 6))


def test_global_vector_kernel_rows_in_tensor_memory():
    """The global-vector kernel on few CTAs (several parts per CTA, rows in
    tensor memory and streamed rows alternating) against the default engine:
    the same solutions to the solver's tolerance."""
    from cbs3d import cases
    gpu = _gpu()
    case = cases.cavity(33, re=400.0, ntime=10 ** 6, jitter=0.15, seed=1234)
    a = gpu.Context(case)
    a.step(2)
    for blocks in (1, 3, 50):
        b = gpu.Context(case, pcg_kernel=5, pcg_blocks=blocks)
        assert b.step(2).pcg_kernel == 8
        assert rel_l2(b.fields()[1], a.fields()[1]) <= 1e-8
        b.close()


# one CTA; two; a few; the largest cluster (16 CTAs, one row per thread)
@pytest.mark.parametrize("n,ctas", [(2, 1), (7, 1), (8, 2), (13, 6), (19, 16)])
def test_cluster_matches_the_grid_of_the_same_ctas(n, ctas):
    """A mesh that fits one thread-block cluster is solved there, exchanging
    through shared memory; a grid of as many CTAs that exchanges through L2
    makes the same sums in the same order."""
    from cbs3d import cases
    gpu = _gpu()
    case = cases.cavity(n, re=400.0, ntime=10 ** 6, jitter=0.15 if n > 2 else 0.0, seed=1234)
    a, b = gpu.Context(case), gpu.Context(case, pcg_kernel=4, pcg_blocks=ctas)
    sa, sb = a.step(3), b.step(3)
    assert sa.cg_iterations_total == sb.cg_iterations_total
    assert sa.cg.final_max_abs == sb.cg.final_max_abs
    for x, y in zip(a.fields(), b.fields()):
        assert bitwise(x, y)


def test_cluster_with_fixed_and_inactive_rows():
    from cbs3d import cases
    gpu = _gpu()
    for case, ctas in ((cases.channel(21, 5, 6, ntime=10 ** 6), 2), (cases.cht_slab(17, 6, 3, 5, ntime=10 ** 6), 3)):
        a, b = gpu.Context(case), gpu.Context(case, pcg_kernel=4, pcg_blocks=ctas)
        a.step(2)
        b.step(2)
        for x, y in zip(a.fields(), b.fields()):
            assert bitwise(x, y)


@pytest.mark.parametrize("rows,spread", [(1, True), (4, False), (8, False)])
def test_batch_tilings_with_a_large_instance(rows, spread):
    """Waves of 512-thread CTAs at one, several and the most rows per thread
    (a tiling whose CTAs do not fit takes the 256-thread kernels): every
    instance as on its own, to the solves' tolerance."""
    from cbs3d import cases
    gpu = _gpu()
    cs = [cases.cavity(n, re=100.0, ntime=10 ** 6) for n in (30, 5, 14)]
    b = gpu.Batch(cs, autotune=False, rows_per_thread=rows, spread=spread)
    bst, _ = b.step(2)
    for i, c in enumerate(cs):
        x = gpu.Context(c)
        st = x.step(2)
        assert abs(bst[i].cg.iterations - st.cg.iterations) <= 2
        for p, q in zip(b.fields(i)[:2], x.fields()[:2]):
            assert rel_l2(p, q) <= 1e-8
        x.close()


def test_two_level_kernel_at_eight_rows_per_thread():
    """The two-level kernel on a uniform mesh, where its layout is larger than
    the single-reduction kernel's: the Jacobi engine's pressure to the solves'
    tolerance, in far fewer iterations."""
    from cbs3d import cases
    gpu = _gpu()
    case = cases.cavity(74, re=400.0, ntime=10 ** 6)
    a, b = gpu.Context(case, two_level=True), gpu.Context(case)
    sa, sb = a.step(1), b.step(1)
    assert sa.pcg_kernel == 6
    assert sa.cg.iterations < sb.cg.iterations
    assert rel_l2(a.fields()[1], b.fields()[1]) <= 1e-8


def test_thin_channel_stays_on_the_register_kernel():
    """A long channel's halos are mostly remote: their state is read from
    global memory, row by row the operations of the global-vector kernel."""
    from cbs3d import cases
    _same(cases.channel(900, 16, 16, length=56.0, ntime=10 ** 6), steps=1)


# tetrahedra between random nodes, so that nearly all columns are remote: about
# 13, 9 and 6 neighbours at one, two and three rows per thread; the box in
# breadth-first order at four
@pytest.mark.parametrize("rows,tets_per_node", [(1, 4.5), (2, 3.0), (3, 2.0), (4, None)])
def test_remote_entries_in_global_memory(rows, tets_per_node):
    """The solved pressure against the operator restated here: the residual is
    the solve's 1e-10 and rounding (well-conditioned operators, sums of 1e5)."""
    from cbs3d import cases
    from test_pcg_partition import partition
    gpu = _gpu()
    rng = np.random.default_rng(rows)
    if tets_per_node is None:
        mesh = cases.box_mesh(64, 64, 64)
    else:
        n = 148 * 512 * rows - 4000
        nodes = np.concatenate([rng.permutation(n) for _ in range(int(np.ceil(tets_per_node)))])
        intma = nodes[:int(n * tets_per_node / 4) * 4].reshape(-1, 4)
        intma = np.concatenate([intma, [[n - 1, 0, 1, 2]]])
        intma = intma[[len(set(t)) == 4 for t in intma.tolist()]]
        mesh = cases.Mesh(coord=np.zeros((n, 3)), intma=(intma + 1).astype(np.int32), bfaces=None, lattice=None, shape=())
    assert partition(mesh, 148, coord=False).single_form == 1
    it, n = mesh.intma - 1, mesh.npoin
    w = -rng.uniform(0.5, 1.5, (it.shape[0], 6))
    pairs = ((0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3))
    diag = np.ones(n)
    for k, (a, b) in enumerate(pairs):
        diag -= np.bincount(it[:, a], w[:, k], n) + np.bincount(it[:, b], w[:, k], n)
    rhs = rng.standard_normal(n)
    solver = gpu.PressureSolver(mesh.intma, None, np.array([1]), np.array([0.0]))
    for _ in range(2):
        x, _, _, res = solver.solve(w, diag, rhs, np.zeros(n))
        assert res["status"] == 0 and res["iterations"] > 5
        r = rhs - diag * x
        for k, (a, b) in enumerate(pairs):
            r -= np.bincount(it[:, a], w[:, k] * x[it[:, b]], n) + np.bincount(it[:, b], w[:, k] * x[it[:, a]], n)
        assert x[0] == 0.0
        assert np.linalg.norm(r[1:]) <= 1e-9 * np.linalg.norm(rhs)
    solver.close()


def test_global_vector_kernel_takes_one_more_part_for_its_slice_table():
    """Two CTAs for 49^3: six halo parts per CTA fit shared memory, but not
    with the table of its 1,954 slices, so it takes seven."""
    from cbs3d import cases
    gpu = _gpu()
    case = cases.cavity(49, re=400.0, ntime=10 ** 6, jitter=0.15, seed=1234)
    a, b = gpu.Context(case), gpu.Context(case, pcg_kernel=5, pcg_blocks=2)
    a.step(1)
    assert b.step(1).pcg_kernel == 8
    assert rel_l2(b.fields()[1], a.fields()[1]) <= 1e-8


# the first and the last size of six rows per thread on 148 SMs
@pytest.mark.parametrize("n", [72, 75])
def test_six_rows_match_the_global_vector_kernel(n):
    from cbs3d import cases
    _same(cases.cavity(n, re=400.0, ntime=10 ** 6, jitter=0.15, seed=1234), steps=1)


# rows of 26 neighbours (centred boxes: one row per thread, two in tensor
# memory, three to five streamed) and of 18 (three in tensor memory, four
# streamed): past the 16 slots that registers and requests hold
@pytest.mark.parametrize("box,n", [("centred_box", 4), ("centred_box", 16), ("centred_box", 28), ("centred_box", 33),
                                   ("centred_box", 37), ("centred_box", 40), ("five_tet_box", 58), ("five_tet_box", 64)])
def test_wide_rows_match_the_global_vector_kernel(box, n):
    import meshes
    _same(meshes.cavity(getattr(meshes, box)(n, n, n)), steps=1)


@pytest.mark.parametrize("n,ctas", [(2, 1), (6, 3), (10, 11)])
def test_cluster_with_wide_rows(n, ctas):
    import meshes
    gpu = _gpu()
    case = meshes.cavity(meshes.centred_box(n, n, n))
    a, b = gpu.Context(case), gpu.Context(case, pcg_kernel=4, pcg_blocks=ctas)
    sa, sb = a.step(2), b.step(2)
    assert sa.cg_iterations_total == sb.cg_iterations_total
    for x, y in zip(a.fields(), b.fields()):
        assert bitwise(x, y)


def test_batch_with_wide_rows():
    import meshes
    gpu = _gpu()
    cs = [meshes.cavity(meshes.centred_box(n, n, n), re=100.0) for n in (12, 3, 17)]
    for rows, spread in ((4, True), (4, False)):
        b = gpu.Batch(cs, autotune=False, rows_per_thread=rows, spread=spread)
        b.step(2)
        for i, c in enumerate(cs):
            x = gpu.Context(c)
            x.step(2)
            for p, q in zip(b.fields(i)[:2], x.fields()[:2]):
                assert rel_l2(p, q) <= 1e-8
            x.close()
        b.close()


@pytest.mark.parametrize("option,n", [("mixed", 70), ("mixed", 76), ("two_level", 76), ("two_level", 20)])
def test_options_that_do_not_fit_run_the_plain_engine(option, n):
    """Where the mixed-precision or the two-level kernel does not fit the mesh
    (too many rows per CTA, or too few), the solve is the Jacobi engine's."""
    from cbs3d import cases
    gpu = _gpu()
    case = cases.cavity(n, re=400.0, ntime=10 ** 6, jitter=0.15, seed=1234)
    a = gpu.Context(case)
    b = gpu.Context(case, precision=gpu.MIXED) if option == "mixed" else gpu.Context(case, two_level=True)
    assert a.step(1).pcg_kernel == b.step(1).pcg_kernel
    for x, y in zip(a.fields(), b.fields()):
        assert bitwise(x, y)


def test_large_batch_with_wide_rows():
    """Four rows per thread of 26 neighbours, which tensor memory does not
    hold, on CTAs of 512 threads."""
    import meshes
    gpu = _gpu()
    cs = [meshes.cavity(meshes.centred_box(n, n, n), re=100.0) for n in (30, 27)]
    b = gpu.Batch(cs, autotune=False)
    b.step(1)
    for i, c in enumerate(cs):
        x = gpu.Context(c)
        x.step(1)
        for p, q in zip(b.fields(i)[:2], x.fields()[:2]):
            assert rel_l2(p, q) <= 1e-8
        x.close()
