"""Results that do not depend on what a context ran before: scratch fields
that a solve leaves behind or starts from, time steps recorded before a call
that changes what they hold, and phase times on every route."""
import numpy as np
import pytest

import iblgf_b200 as B
import iblgf_setups as S
import oracle_lib as O

pytestmark = pytest.mark.gpu


def solver(case, **kw):
    return B.Solver(case.bd_base, case.bd_extent, case.block_extent, case.dx_base, case.blocks,
                    n_levels=case.n_levels, predicate=case.predicate, **kw)


def ring(g, case):
    u = case.initial_velocity(g)
    return [g.field(u[k]) for k in range(3)], g.field()


@pytest.mark.parametrize("route", ["replayed step", "recorded solve", "pointer"])
def test_stream_solve_clears_correction(route):
    """A solve without a source correction leaves correction_tmp zero (PoissonSolver::apply_lgf cleans it first),
    whoever wrote it since the last such solve."""
    torch = pytest.importorskip("torch")
    case = S.VortexRingNS("small")
    stream = torch.cuda.Stream()
    g = solver(case, stream=stream.cuda_stream)
    uf, pf = ring(g, case)
    T = g.ns_step(uf, pf, case.dt(), case.Re, 0.0, 3)  # direct, recorded, replayed
    corr = g.ns_fields()[2]
    rng = np.random.default_rng(2)
    fs, ft = g.field(rng.standard_normal((g.n, g.Nb, g.Nb, g.Nb))), g.field()
    ptr = g.device_ptr(corr)
    graph = torch.cuda.CUDAGraph()
    if route == "recorded solve":
        g.apply_lgf(fs, ft)
        g.synchronize()
        with torch.cuda.graph(graph, stream=stream):
            g.apply_lgf(fs, ft)
    g.apply_lgf(fs, ft, B.STREAM)
    assert not g.download(corr).any()
    g.apply_lgf(fs, ft, B.STREAM)  # finds the field clean
    g.synchronize()
    if route == "replayed step":
        g.ns_step(uf, pf, case.dt(), case.Re, T, 1)
    elif route == "recorded solve":
        graph.replay()
    else:
        view = type("View", (), {"__cuda_array_interface__": {"shape": (g.n * g.Nb ** 3,), "typestr": "<f8",
                                                              "data": (ptr, False), "version": 2}})()
        torch.as_tensor(view, device="cuda").fill_(1.0)
    torch.cuda.synchronize()
    g.apply_lgf(fs, ft, B.STREAM)
    assert not g.download(corr).any()


def test_octants_without_a_parent():
    """An imported octant list may leave out an octant whose children it has: no interpolation writes these
    children, and every solve starts them from zero."""
    e = 6
    args = ((-4 * e,) * 3, (8 * e,) * 3, e, 0.5, [((-2 * e,) * 3, (4 * e,) * 3)])
    whole = B.Solver(*args, n_levels=1, predicate=lambda base, ext, rl, diff: rl == 0 and tuple(base) == (0, 0, 0))
    refined = [o for o in range(whole.n) if whole.levels[o] == whole.base_level and not whole.flags[o] & 3]
    assert refined
    keep = np.array([o not in refined for o in range(whole.n)])
    imp = (whole.keys[keep], whole.flags[keep])
    rng = np.random.default_rng(4)
    a, b = rng.standard_normal((2, int(keep.sum()), e + 2, e + 2, e + 2))
    out = []
    for first in (None, a):
        g = B.Solver(*args, import_octants=imp)
        assert np.any((g.levels == g.base_level + 1) & (g.flags & 1))
        fs, ft = g.field(), g.field()
        for x in (first, b):
            if x is None:
                continue
            g.upload(fs, x)
            g.apply_lgf(fs, ft)
        out.append(g.download(ft))
    assert out[0].any()
    np.testing.assert_array_equal(out[1], out[0])


@pytest.mark.parametrize("direct", [True, False])
def test_integrating_factor_phase_times(direct):
    """iblgf_profile_read covers the integrating factor's sums on both of its routes."""
    case = S.VortexRingNS("small")
    g = solver(case)
    g.ge_direct(direct)
    fs, ft = g.field(np.ones((g.n, g.Nb, g.Nb, g.Nb))), g.field()
    g.apply_if(fs, ft, 1e-3)
    g.profile(True)
    g.apply_if(fs, ft, 1e-3)
    assert g.profile_read()[2] > 0


@pytest.mark.parametrize("call", ["apply_if", "stream", "refresh", "points", "ge_direct", "cg", "warmstart"])
def test_step_after_another_call(call):
    """A recorded step is not replayed over memory that a later call replaced (a kernel table, spectra and work
    buffers of a sweep that was not there before, the immersed-boundary points), nor past a switch that a later call
    set. Against a context that launches every step directly (it takes phase times), bit for bit with the same MAC
    variant."""
    ib = call in ("points", "cg", "warmstart")
    case = S.SphereIB("small") if ib else S.VortexRingNS("small")
    out = []
    for direct in (False, True):
        g = solver(case)
        g.mac_variant(0)
        if ib:
            X = O.sphere_points(case.dx_base, g.depth - 1 - g.base_level, case.ibph)
            g.ib_set_points(X, case.Re)
            g.ns_options((-1.0, 0.0, 0.0))
            u, dt = case.velocity(g), 0.01
        else:
            u, dt = case.initial_velocity(g), case.dt()
        uf, pf = [g.field(u[k]) for k in range(3)], g.field()
        g.profile(direct)
        T = g.ns_step(uf, pf, dt, case.Re, 0.0, 3)  # direct, recorded, replayed
        fs, ft = g.field(u[0]), g.field()
        if call == "apply_if":
            for k in range(20):
                g.apply_if(fs, ft, 0.01 + 1e-3 * k)
        elif call == "stream":
            g.apply_lgf(fs, ft, B.STREAM)
        elif call == "refresh":
            T = g.ns_step(uf, pf, dt, case.Re, T + 1e6, 1)
        elif call == "points":
            g.ib_set_points(X[: len(X) // 2], case.Re)
        elif call == "ge_direct":
            g.ge_direct(False)
        elif call == "cg":
            g.ns_options((-1.0, 0.0, 0.0), cg_threshold=1e-8)
        else:
            g.ib_warmstart(2)
        g.ns_step(uf, pf, dt, case.Re, T, 3)
        out.append(np.stack([g.download(f) for f in uf + [pf]]))
    assert out[0].any()
    np.testing.assert_array_equal(out[0], out[1])
