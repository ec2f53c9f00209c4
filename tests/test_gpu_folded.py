"""M2L folded over mirrored offsets (m2l_sym.cu), the r = 32 kernels (m2l_r32.cu) and the heavy
leaves of P2M / L2P, against the oracle (-m gpu).

Tolerances: FP64 1e-12 (order of the sums; measured 1e-15 class), FP32 2e-5 (as the parity tests of
the FP32 solve), mixed 3e-7 against FP64 (the split products' rounding, measured 4e-8)."""
import numpy as np
import pytest

from conftest import uniform_inputs
from oracle.oracle import Oracle, rel_l2

pytestmark = pytest.mark.gpu


def _ops(n, single=False, kernel="laplacian"):
    from bbfmm_b200 import operators as ops
    _, U, E = ops.load_operators(n, single=single, kernel=kernel)
    return np.asarray(U), np.asarray(E)


def _solve(x, q, n, lev, mode, U, E, **kw):
    import torch
    from bbfmm_b200 import Solver
    s = Solver(n, lev, 1.0, mode=mode, operators=(U, E), **kw)
    s.set_particles(x)
    out = s.solve(torch.as_tensor(q, dtype=s.dtype, device="cuda")).double().cpu().numpy()
    return s, out


@pytest.mark.parametrize("n", [4, 8])
@pytest.mark.parametrize("lev", [2, 3, 4])
def test_levels_match_the_oracle(n, lev):
    """Every level's tile form (stacked 2 x 2 x 2 grids, one box, many boxes), FP64 and FP32."""
    x, q = uniform_inputs(3001, seed=10 * n + lev)
    U, E = _ops(n)
    ref = Oracle("d").fmm(x, q, n, lev, U, E)
    s, got = _solve(x, q, n, lev, "d", U, E)
    assert rel_l2(got, ref) < 1e-12
    tree = Oracle("d").build_tree(x, lev)
    _, P = Oracle("d").upward(tree, x, q, n, U)
    r = n ** 3 // 2
    for l in range(2, lev + 1):  # in the basis of the operators as given
        lo = (8 ** l - 1) // 7
        assert rel_l2(s.multipoles(l), P[lo * r:(lo + 8 ** l) * r]) < 1e-13
    s.close()
    Us, Es = _ops(n, single=True)
    s, got = _solve(x, q, n, lev, "s", Us, Es)
    assert rel_l2(got, ref) < 2e-5
    s.close()


@pytest.mark.parametrize("mode", ["d", "s", "mixed"])
@pytest.mark.parametrize("sets", [1, 7, 8, 9, 17])
def test_stacked_sets(mode, sets):
    """Sets stacked at levels 2 and 3: counts around the eight sets of a level-2 tile."""
    import torch
    from bbfmm_b200 import Batch, Solver
    rng = np.random.default_rng(sets)
    xs = [rng.random((50 + 13 * k, 3)) - 0.5 for k in range(sets)]
    b = Batch([(x, n, 3) for x in xs for n in (4, 8)], mode=mode)
    q = rng.uniform(-1, 1, b.N)
    got = b.solve(torch.as_tensor(q, dtype=b.dtype, device="cuda")).double().cpu().numpy()
    b.close()
    for n in (4, 8):
        s = Solver(n, 3, 1.0, mode="d")
        for k, x in enumerate(xs):
            i = 2 * k + (n == 8)
            a, e = int(b.offsets[i]), int(b.offsets[i + 1])
            s.set_particles(x)
            want = s.solve(torch.as_tensor(q[a:e], device="cuda")).cpu().numpy()
            assert rel_l2(got[a:e], want) < {"d": 1e-12, "s": 2e-5, "mixed": 3e-7}[mode]
        s.close()


def test_any_basis_of_the_same_span():
    """U Q and Q^T E Q for a random orthogonal Q: the same potentials (the rotation that sorts the
    components by parity starts from whatever basis is given)."""
    n, lev, r, n3 = 8, 3, 256, 512
    U, E = _ops(n)
    Q, _ = np.linalg.qr(np.random.default_rng(1).standard_normal((r, r)))
    U2 = (U.reshape(r, n3).T @ Q).T.reshape(-1)
    Ek = E.reshape(316, r, r).transpose(0, 2, 1)
    E2 = (Q.T @ Ek @ Q).transpose(0, 2, 1).reshape(-1)
    x, q = uniform_inputs(4000, seed=3)
    s, a = _solve(x, q, n, lev, "d", U, E)
    s.close()
    s, b = _solve(x, q, n, lev, "d", np.ascontiguousarray(U2), np.ascontiguousarray(E2))
    s.close()
    # the products that make U2 and E2 round at 1e-15 of their largest entries
    assert rel_l2(b, a) < 1e-11


def test_operators_without_the_symmetry_take_the_general_path():
    """One offset's operator changed: the images no longer agree, and the solve follows the given
    operators all the same."""
    n, lev, r = 8, 3, 256
    U, E = _ops(n)
    E = E.copy()
    E[5 * r * r:6 * r * r] *= 1.5
    x, q = uniform_inputs(3000, seed=4)
    ref = Oracle("d").fmm(x, q, n, lev, U, E)
    s, got = _solve(x, q, n, lev, "d", U, E)
    assert rel_l2(got, ref) < 1e-12
    s.close()


@pytest.mark.parametrize("count", [63, 64, 65, 128, 129, 1000])
@pytest.mark.parametrize("n,mode", [(4, "d"), (8, "d"), (4, "s"), (8, "mixed")])
def test_heavy_leaves(count, n, mode):
    """Leaves around the cap of 64 particles a warp takes: P2M chunks, their join, L2P chunks."""
    import torch
    rng = np.random.default_rng(count)
    x = np.concatenate([rng.random((count, 3)) * 0.12 - 0.5, rng.random((count // 2, 3)) * 0.12 + 0.26,
                        rng.random((200, 3)) - 0.5])
    q = rng.uniform(-1, 1, len(x))
    U, E = _ops(n)
    ref = Oracle("d").fmm(x, q, n, 3, U, E)
    Um, Em = _ops(n, single=mode == "s")
    s, got = _solve(x, q, n, 3, mode, Um, Em)
    assert rel_l2(got, ref) < {"d": 1e-12, "s": 2e-5, "mixed": 3e-7}[mode]
    pot, fld = s.solve_fields(torch.as_tensor(q, dtype=s.dtype, device="cuda"))
    assert rel_l2(pot.double().cpu().numpy() * q, ref) < {"d": 1e-12, "s": 2e-5, "mixed": 3e-7}[mode]
    s.close()


@pytest.mark.parametrize("lev,sets", [(2, 33), (3, 5), (3, 9), (4, 1), (4, 3)])
def test_offset_groups_of_small_tensor_core_levels(lev, sets):
    """Levels of a few tensor-core tiles split their offsets over CTAs: nine groups, fewer where
    stacked sets fill more tiles (a partial last tile, an odd count of tiles per class)."""
    import torch
    from bbfmm_b200 import Batch
    rng = np.random.default_rng(100 * lev + sets)
    xs = [rng.random((300 * 2 ** (lev - 2) + 7 * k, 3)) - 0.5 for k in range(sets)]
    out = {}
    for mode in ("mixed", "d"):
        b = Batch([(x, 8, lev) for x in xs], mode=mode)
        q = np.random.default_rng(5).uniform(-1, 1, b.N)
        out[mode] = b.solve(torch.as_tensor(q, device="cuda")).cpu().numpy()
        off = b.offsets
        b.close()
    for k in range(sets):
        a, e = int(off[k]), int(off[k + 1])
        assert rel_l2(out["mixed"][a:e], out["d"][a:e]) < 3e-7


def _after_a_change(s, q, level, change):
    """multipoles() and m2l_output() of a level before and after `change` and a timing call, with no
    solve in between."""
    import torch
    s.solve(torch.as_tensor(q, dtype=s.dtype, device="cuda"))
    before = s.multipoles(level), s.m2l_output(level)
    change()
    s.time_m2l(level, 1)
    return before, (s.multipoles(level), s.m2l_output(level))


@pytest.mark.parametrize("level,kinds", [(3, (0, 2)), (3, (2, 0)), (4, (0, 1)), (4, (1, 0))])
def test_read_back_after_a_change_of_the_m2l_kind(level, kinds):
    """Mixed mode, a level moved between the folded FP64 M2L and the tensor cores: the multipoles
    stay those of the solve (1e-13: one rotation to the operators' basis) and the M2L output is
    theirs under either kind (1e-6, the tolerance of the tensor-core M2L elsewhere)."""
    from bbfmm_b200 import Solver
    x, q = uniform_inputs(3000, seed=level)
    s = Solver(8, 4, 1.0, mode="mixed")

    def kind(k):
        t = s.tuning()
        t["m2l_kind"][level] = k
        s.set_tuning(t)

    kind(kinds[0])
    s.set_particles(x)
    (m0, l0), (m1, l1) = _after_a_change(s, q, level, lambda: kind(kinds[1]))
    assert rel_l2(m1, m0) < 1e-13
    assert rel_l2(l1.ravel(), l0.ravel()) < 1e-6
    s.close()


@pytest.mark.parametrize("mode", ["d", "s"])
@pytest.mark.parametrize("ranks", [(0, 160), (160, 0)])
def test_read_back_after_a_change_of_the_rank(mode, ranks):
    """The rank set (which takes the unfolded kernel, components below it) or cleared after the
    solve: the multipoles stay, and the M2L output is that of the rank in force."""
    from bbfmm_b200 import _lib
    from bbfmm_b200 import operators as ops
    level, r = 3, 256
    x, q = uniform_inputs(3000, seed=9)
    U, E = _ops(8, single=mode == "s")
    from bbfmm_b200 import Solver
    s = Solver(8, 3, 1.0, mode=mode, operators=(U, E))
    rank = lambda k: _lib.check(_lib.lib().bbfmm_b200_set_rank(s.h, k))
    rank(ranks[0])
    s.set_particles(x)
    (m0, _), (m1, l1) = _after_a_change(s, q, level, lambda: rank(ranks[1]))
    tol = 1e-12 if mode == "d" else 2e-5
    assert rel_l2(m1.astype(float), m0.astype(float)) < (1e-13 if mode == "d" else 1e-6)
    k = ranks[1] or r
    if k != r:
        U, E = ops.truncate_operators(8, U, E, k)
    cells = np.arange(0, 8 ** level, 37)
    want = Oracle("d").m2l_sample(level, r, E.astype(float), m1.astype(float), cells)
    assert rel_l2(l1[cells][:, :k].astype(float).ravel(), np.asarray(want).reshape(len(cells), r)[:, :k].ravel()) < tol
    s.close()


def test_autotune_leaves_the_multipoles_in_the_given_basis():
    import torch
    from bbfmm_b200 import Solver
    x, q = uniform_inputs(4000, seed=2)
    s = Solver(8, 4, 1.0, mode="mixed")
    s.set_particles(x)
    s.solve(torch.as_tensor(q, dtype=s.dtype, device="cuda"))
    want = [s.multipoles(l) for l in (2, 3, 4)]
    s.autotune(torch.as_tensor(q, dtype=s.dtype, device="cuda"))
    for l, w in zip((2, 3, 4), want):
        assert rel_l2(s.multipoles(l), w) < 3e-7
    s.close()


def _forms(n, mode, lev=4, operators=None, **kw):
    from bbfmm_b200 import Solver
    s = Solver(n, lev, 1.0, mode=mode, operators=operators, **kw)
    f = [s.m2l_form(l) for l in range(2, lev + 1)]
    s.close()
    return f


def test_the_form_of_the_m2l():
    """Which M2L runs: the tests above pass on the dense kernels too, so the form is stated here."""
    assert _forms(8, "d") == _forms(8, "s") == ["folded"] * 3
    assert _forms(8, "mixed") == ["folded", "folded", "tensor"]
    for mode in ("d", "s", "mixed"):
        assert _forms(4, mode) == ["r32"] * 3
    # a rank cut, kernels odd in an axis or with a basis of mixed parity
    assert _forms(8, "d", rank=128) == ["dense"] * 3
    for kernel in ("laplacianforce", "oneoverr4"):
        assert _forms(8, "d", kernel=kernel) == ["dense"] * 3


def test_the_form_of_other_operators():
    """The rotated basis of test_any_basis_of_the_same_span is folded, the operator changed in
    test_operators_without_the_symmetry_take_the_general_path is not."""
    r, n3 = 256, 512
    U, E = _ops(8)
    Q, _ = np.linalg.qr(np.random.default_rng(1).standard_normal((r, r)))
    U2 = np.ascontiguousarray((U.reshape(r, n3).T @ Q).T.reshape(-1))
    E2 = np.ascontiguousarray((Q.T @ E.reshape(316, r, r).transpose(0, 2, 1) @ Q).transpose(0, 2, 1).reshape(-1))
    assert _forms(8, "d", operators=(U2, E2)) == ["folded"] * 3
    E = E.copy()
    E[5 * r * r:6 * r * r] *= 1.5
    assert _forms(8, "d", operators=(U, E)) == ["dense"] * 3


def _output_by_components(U, E, mode):
    """The M2L output of level 3 against the oracle's from the same multipoles and operators, per 64
    components (their operators fall from 1 to 1e-10 of the largest entry): relative errors."""
    import torch
    from bbfmm_b200 import Solver
    x, q = uniform_inputs(3000, seed=6)
    s = Solver(8, 3, 1.0, mode=mode, operators=(U, E))
    form = s.m2l_form(3)
    s.set_particles(x)
    s.solve(torch.as_tensor(q, dtype=s.dtype, device="cuda"))
    cells = np.arange(0, 512, 5)
    got = s.m2l_output(3)[cells].astype(float)
    want = Oracle("d").m2l_sample(3, 256, np.asarray(E, float), s.multipoles(3).astype(float), cells).reshape(-1, 256)
    s.close()
    return form, [rel_l2(got[:, a:a + 64].ravel(), want[:, a:a + 64].ravel()) for a in range(0, 256, 64)]


# components of FP32 output are rounded and summed as those of the solve (2e-5); in FP64 the folded
# operators are off the given ones by at most 64 roundings (7e-15) of the largest entry, against
# entries of 1e-3, 1e-6, 2e-8 and 1e-9 of it
BY_COMPONENT = {"s": [2e-5] * 4, "d": [1e-11, 1e-8, 1e-6, 1e-5]}


@pytest.mark.parametrize("mode", ["d", "s"])
def test_high_components_keep_their_precision(mode):
    U, E = _ops(8, single=mode == "s")
    form, err = _output_by_components(U, E, mode)
    assert form == "folded"
    assert all(e < t for e, t in zip(err, BY_COMPONENT[mode])), err


@pytest.mark.parametrize("mode,rows,factor", [("s", 64, 1.5), ("s", 128, 1.01), ("s", 192, 1.01), ("d", 128, 1.001),
                                              ("d", 240, 1.001)])
def test_operators_that_differ_beyond_their_rounding_are_not_folded(mode, rows, factor):
    """The high components of one offset's operator changed: far below a rounding of the largest
    entry, and the M2L still follows the operators given."""
    U, E = _ops(8, single=mode == "s")
    E = E.reshape(316, 256, 256).copy()
    k = 202  # offset (1, 1, 2)
    E[k, :, rows:] *= E.dtype.type(factor)
    form, err = _output_by_components(U, E.reshape(-1), mode)
    assert form == "dense"
    assert max(err) < (2e-5 if mode == "s" else 1e-12), err


@pytest.mark.parametrize("mode", ["d", "s"])
def test_operators_that_differ_by_their_rounding_are_folded(mode):
    """Every entry changed by up to two roundings of its own."""
    U, E = _ops(8, single=mode == "s")
    u = np.finfo(E.dtype).eps / 2
    E2 = (E * (1 + 2 * u * np.random.default_rng(3).uniform(-1, 1, E.size))).astype(E.dtype)
    form, err = _output_by_components(U, E2, mode)
    assert form == "folded"
    assert all(e < t for e, t in zip(err, BY_COMPONENT[mode])), err


@pytest.mark.parametrize("n", [4, 8])
@pytest.mark.parametrize("level", [2, 3])
def test_fp32_sums_do_not_depend_on_the_groups(n, level):
    """The 189 offsets split over 1 to 21 CTAs: partial sums stay in FP64, so that the FP32 output is
    one rounding of the same sum (a value may fall to the other side of a tie of FP32, about one in
    1e7; one in 1e3 is allowed) and as close to the oracle as that rounding."""
    import torch
    from bbfmm_b200 import Solver
    x, q = uniform_inputs(3000, seed=n + level)
    U, E = _ops(n, single=True)
    s = Solver(n, 3, 1.0, mode="s", operators=(U, E))
    s.set_particles(x)
    out = []
    for g in (1, 2, 7, 21):
        t = s.tuning()
        t["m2l_groups"][level] = g
        s.set_tuning(t)
        if not out:
            s.solve(torch.as_tensor(q, dtype=s.dtype, device="cuda"))
        out.append(s.m2l_output(level))
    for o in out[1:]:
        assert np.mean(o != out[0]) < 1e-3
    if n == 4:  # the multipoles read back are the ones contracted
        r = n ** 3 // 2
        want = Oracle("d").m2l_sample(level, r, E.astype(float), s.multipoles(level).astype(float), np.arange(8 ** level))
        assert rel_l2(out[-1].astype(float).ravel(), np.asarray(want).ravel()) < 2.0 ** -24
    s.close()


def test_a_regions_sums_do_not_depend_on_earlier_tunings():
    """The folded M2L of a target region's block list: its step groups follow from the level and the
    list, whatever scratch an earlier tuning of the same solver left, and the results are the same
    bits; particles in the region agree with the unrestricted solve."""
    import torch
    from bbfmm_b200 import Solver
    from bbfmm_b200.fmm import leaf_of_particles
    x, q = uniform_inputs(20000, seed=8)
    qd = torch.as_tensor(q, device="cuda")
    active = np.zeros(64, bool)
    active[[5, 40]] = True
    inside = active[leaf_of_particles(x, 1.0, 2)[0]]
    got, groups = [], []
    for more in (False, True):
        s = Solver(8, 4, 1.0, mode="d")
        s.set_particles(x)
        if more:
            whole = s.solve(qd).cpu().numpy()
            for g in (21, 0):
                t = s.tuning()
                t["m2l_groups"] = [g] * 11
                s.set_tuning(t)
        s.set_target_region(2, active)
        got.append(s.solve(qd).cpu().numpy()[inside])
        groups.append([s.m2l_groups(l) for l in (2, 3, 4)])
        s.close()
    assert groups[0] == groups[1]
    assert groups[0][2] == 16  # a list of two blocks at level 4: 18 would fill the GPU, 16 slices is the bound
    assert np.array_equal(got[0], got[1])
    assert rel_l2(got[0], whole[inside]) < 1e-12


@pytest.mark.parametrize("mode,change", [("d", "rank"), ("mixed", "products")])
def test_choices_after_the_particles_get_their_scratch(mode, change):
    """The rank or the products set after the particles: the groups that they take before them."""
    from bbfmm_b200 import Solver, _lib
    x, _ = uniform_inputs(3000, seed=1)
    lev = 3 if change == "rank" else 4  # depths at which the first choice's scratch is the smaller
    groups = []
    for late in (False, True):
        s = Solver(8, lev, 1.0, mode=mode)
        if change == "products":
            s.set_tc_products(3)
        if late:
            s.set_particles(x)
        if change == "rank":
            _lib.check(_lib.lib().bbfmm_b200_set_rank(s.h, 160))
        else:
            s.set_tc_products(0)
        if not late:
            s.set_particles(x)
        groups.append([s.m2l_groups(l) for l in range(2, lev + 1)])
        s.close()
    assert groups[0] == groups[1] and max(groups[0]) > 1


def test_the_near_list_keeps_no_scratch():
    """Device memory that a particle more costs at one depth: its FP32 position, charge and potential,
    an index and 8 bytes of the list (32 bytes), and no scratch of the list's order (8 more)."""
    import torch
    from bbfmm_b200 import Solver
    used = []
    rng = np.random.default_rng(0)
    for N in (1_000_000, 9_000_000):
        s = Solver(4, 4, 1.0, mode="s")
        x = torch.as_tensor(rng.random((N, 3)) - 0.5, dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        s.set_particles(x)
        used.append(free - torch.cuda.mem_get_info()[0])
        s.close()
        del x
    assert 30 < (used[1] - used[0]) / 8e6 < 34


@pytest.mark.parametrize("mode", ["d", "mixed"])
def test_the_rotation_of_the_operators_needs_little_memory(mode):
    """Device memory that the creation of an n = 8 solver holds for a time, above what it keeps
    (sampled beside it): below 200 MB, of which the mixed mode's own set-up takes some."""
    import threading
    import torch
    from bbfmm_b200 import Solver
    U, E = _ops(8)
    Solver(8, 3, 1.0, mode=mode, operators=(U, E)).close()  # context and modules
    free, done = [], threading.Event()

    def sample():
        while not done.is_set():
            free.append(torch.cuda.mem_get_info()[0])

    t = threading.Thread(target=sample)
    t.start()
    s = Solver(8, 3, 1.0, mode=mode, operators=(U, E))
    done.set()
    t.join()
    assert s.m2l_form(3) == "folded"
    kept = torch.cuda.mem_get_info()[0]
    s.close()
    assert len(free) > 10 and kept - min(free) < 200e6, (kept - min(free), len(free))
