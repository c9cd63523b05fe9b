"""Results that do not depend on what a context ran before: scratch fields
that a solve leaves behind."""
import numpy as np
import pytest

import iblgf_b200 as B
import iblgf_setups as S

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
