"""Block kernels over the block extents and the edges of their work splits,
against the oracle: sweeps with partly present sibling groups, the integrating
factor's truncation radii, the single-block convolution, the Fourier-in-z
operators at extents without a compile-time form, interpolation orders, both
forms of the anterpolation, and few immersed-boundary points."""
import os
import sys

import numpy as np
import pytest

import iblgf_b200 as B
import iblgf_setups as S
import oracle_lib as O

sys.path.insert(0, os.path.join(os.path.dirname(__file__), "..", "oracle"))
import helm2d as H  # noqa: E402

pytestmark = pytest.mark.gpu


def rel_linf(a, b):
    return float(np.abs(a - b).max() / max(np.abs(b).max(), 1e-300))


def uneven(e, precision, **kw):
    """3 x 2 x 1 base blocks (groups with 1, 2 and 4 of their 8 blocks, an odd number of groups), the block at the
    origin refined once."""
    args = ((-4 * e,) * 3, (8 * e,) * 3, e, 0.5, [((-2 * e, -e, 0), (3 * e, 2 * e, e))])
    pred = lambda base, ext, rl, diff: rl == 0 and tuple(base) == (0, 0, 0)  # noqa: E731
    return (O.Domain(*args, n_levels=1, predicate=pred),
            B.Solver(*args, n_levels=1, predicate=pred, precision=precision, **kw))


@pytest.mark.parametrize("variant", [0, 1])
@pytest.mark.parametrize("precision,tol", [(B.FP64, 1e-12), (B.FP32, 1e-5)])
@pytest.mark.parametrize("e", [4, 6, 8, 10, 14, 16])
def test_solve_uneven_octree(e, precision, tol, variant):
    """apply_lgf with both shapes of the direct MAC, twice on the same context (the second from scratch fields that
    the first has filled); tolerances: the FP64 and FP32 parity bars."""
    o, g = uneven(e, precision)
    g.mac_variant(variant)
    src = np.random.default_rng(e).standard_normal((o.n, o.Nb, o.Nb, o.Nb))
    ref = o.apply_lgf(src)
    fs, ft = g.field(src), g.field()
    for _ in range(2):
        g.apply_lgf(fs, ft)
        assert rel_linf(g.download(ft), ref) < tol


# e^{-2a} I_m(2a) falls below 2^-56 of its centre beyond m = 4, 6, 8, 12, 16 for these a
@pytest.mark.parametrize("alpha", [4e-4, 8e-3, 4e-2, 0.25, 0.6])
@pytest.mark.parametrize("e", [4, 10, 16])
def test_integrating_factor_radii(e, alpha):
    """Separable sums and block convolutions against the oracle, into another field and into the source itself."""
    o, g = uneven(e, B.FP64)
    src = np.random.default_rng(e).standard_normal((o.n, o.Nb, o.Nb, o.Nb))
    ref = o.apply_if(src, alpha)
    for direct in (True, False):
        g.ge_direct(direct)
        fs, ft = g.field(src), g.field()
        g.apply_if(fs, ft, alpha)
        assert rel_linf(g.download(ft), ref) < 1e-12
        g.apply_if(fs, fs, alpha)
        sel = np.asarray(o.levels) >= o.base_level  # the coarser blocks keep their values
        assert rel_linf(g.download(fs)[sel], ref[sel]) < 1e-12


@pytest.mark.parametrize("precision,tol", [(B.FP64, 1e-12), (B.FP32, 1e-5)])
@pytest.mark.parametrize("e", [4, 6, 8, 10, 14, 16])
def test_conv_block_extents(e, precision, tol):
    """The single-block convolution adds to its output; twice, so that the kept work buffer is used again."""
    torch = pytest.importorskip("torch")
    N = e + 2
    P = 2 * N - 1
    g = B.Solver((-2 * e,) * 3, (4 * e,) * 3, e, 1.0, [((-e,) * 3, (2 * e,) * 3)], precision=precision)
    rng = np.random.default_rng(e)
    for _ in range(2):
        src, ker = rng.standard_normal((N, N, N)), rng.standard_normal((P, P, P))
        base = rng.standard_normal(N ** 3)
        out = torch.tensor(base, device="cuda")
        ts, tk = (torch.tensor(a.ravel(order="F"), device="cuda") for a in (src, ker))
        torch.cuda.synchronize()
        g.conv_block(ts.data_ptr(), tk.data_ptr(), out.data_ptr(), 0.5)
        ref = O.block_conv(src, ker, 0.5).ravel(order="F")
        assert rel_linf(out.cpu().numpy() - base, ref) < tol


# the 2-norm error is the mean over the block's 512 and 5832 nodes and six inputs, within 2 % from seed to seed; direct
# sums of 15 and 35 terms in the inverse z and y passes give 8.3e-16 at both, the prime-factor sums 7.5e-16 and 7.2e-16
@pytest.mark.parametrize("e,bound", [(6, 7.85e-16), (16, 7.75e-16)])
def test_conv_block_rounding(e, bound):
    """The FP64 convolution against extended precision where P = 2 Nb - 1 splits into coprime factors."""
    torch = pytest.importorskip("torch")
    N, P = e + 2, 2 * e + 3
    g = B.Solver((-2 * e,) * 3, (4 * e,) * 3, e, 1.0, [((-e,) * 3, (2 * e,) * 3)])
    err = []
    for seed in range(6):
        rng = np.random.default_rng(seed)
        src, ker = rng.standard_normal((N, N, N)), rng.standard_normal((P, P, P))
        ref, lk = np.zeros((N, N, N), np.longdouble), ker.astype(np.longdouble)
        for z, y, x in np.ndindex(N, N, N):
            ref += np.longdouble(src[z, y, x]) * lk[N - 1 - z:P - z, N - 1 - y:P - y, N - 1 - x:P - x]
        out = torch.zeros(N ** 3, dtype=torch.float64, device="cuda")
        ts, tk = torch.tensor(src.ravel(), device="cuda"), torch.tensor(ker.ravel(), device="cuda")
        torch.cuda.synchronize()
        g.conv_block(ts.data_ptr(), tk.data_ptr(), out.data_ptr(), 1.0)
        d = out.cpu().numpy().reshape(N, N, N).astype(np.longdouble) - ref
        err.append(float(np.sqrt((d ** 2).sum() / (ref ** 2).sum())))
    assert np.mean(err) < bound, np.mean(err)


@pytest.mark.parametrize("nb,nm", [(3, 1), (7, 5), (18, 7), (40, 3)])
@pytest.mark.parametrize("op", ["laplace", "gradient", "divergence", "curl", "curl_transpose"])
def test_fourier_operators_extents(op, nb, nm):
    """Extents with and without a compile-time form, from less than a CTA's work to several CTAs per block."""
    import torch
    g = B.Solver((-12,) * 3, (24,) * 3, 6, 1.0, [((-6,) * 3, (12,) * 3)])
    rng = np.random.default_rng(nb)
    sep = 2 * nm
    cin = sep if op in ("laplace", "gradient") else 3 * sep
    cout = sep if op in ("laplace", "divergence") else 3 * sep
    src, dst = rng.standard_normal((2, cin, nb, nb)), rng.standard_normal((2, cout, nb, nb))
    ref = H.helm_op(op, src, dst.copy(), nm, 0.25, 1.5, 0.6)
    s, d = torch.tensor(src, device="cuda"), torch.tensor(dst, device="cuda")
    torch.cuda.synchronize()
    g.helm2d_op(op, s, d, nm, 0.25, 1.5, 0.6)
    g.synchronize()
    assert np.abs(d.cpu().numpy() - ref).max() < 1e-13 * np.abs(ref).max()


@pytest.mark.parametrize("nb,npl", [(3, 1), (7, 5), (18, 7), (40, 3)])
def test_fourier_nonlinear_extents(nb, npl):
    """As test_fourier_operators_extents, the collocation-plane convective term; its bar in test_gpu_helm2d.py."""
    import torch
    g = B.Solver((-12,) * 3, (24,) * 3, 6, 1.0, [((-6,) * 3, (12,) * 3)])
    face, edge, dst = np.random.default_rng(nb).standard_normal((3, 2, 3 * npl, nb, nb))
    ref = H.nonlinear(face, edge, dst.copy(), npl, None)
    d = torch.tensor(dst, device="cuda")
    f, e = torch.tensor(face, device="cuda"), torch.tensor(edge, device="cuda")
    torch.cuda.synchronize()
    g.helm2d_nonlinear(f, e, d, npl)
    g.synchronize()
    assert np.abs(d.cpu().numpy() - ref).max() < 1e-14 * np.abs(ref).max()


# band widths of the cell-centred transfers: 2 (orders 1, 2), the window of 5 (3 to 5), dense (above)
@pytest.mark.parametrize("order", [1, 2, 3, 4, 6, 7, 11])
@pytest.mark.parametrize("e", [4, 16])
def test_interpolation_orders(e, order):
    """apply_lgf across a level change; the FP64 parity bar."""
    args = ((-4 * e,) * 3, (8 * e,) * 3, e, 0.5, [((-2 * e, -e, 0), (3 * e, 2 * e, e))])
    kw = dict(n_levels=1, predicate=lambda base, ext, rl, diff: rl == 0 and tuple(base) == (0, 0, 0), intrp_order=order)
    o, g = O.Domain(*args, **kw), B.Solver(*args, **kw)
    src = np.random.default_rng(e).standard_normal((o.n, o.Nb, o.Nb, o.Nb))
    fs, ft = g.field(src), g.field()
    g.apply_lgf(fs, ft)
    assert rel_linf(g.download(ft), o.apply_lgf(src)) < 1e-12


@pytest.mark.parametrize("order", [2, 4, 7])
def test_interpolation_orders_time_step(order):
    """Face and edge fields take two matrix sets per transfer; the bar of the plain time steps (FP64)."""
    case = S.VortexRingNS("small")
    args = (case.bd_base, case.bd_extent, case.block_extent, case.dx_base, case.blocks)
    kw = dict(n_levels=case.n_levels, predicate=case.predicate, intrp_order=order)
    o, g = O.Domain(*args, **kw), B.Solver(*args, **kw)
    u0 = case.initial_velocity(o)
    ur, pr = o.ns_step(u0, case.dt(), case.Re, 0.0, 1)
    uf, pf = [g.field(u0[k]) for k in range(3)], g.field()
    g.ns_step(uf, pf, case.dt(), case.Re, 0.0, 1)
    for f, ref in zip(uf + [pf], list(ur) + [pr]):
        assert rel_linf(g.download(f), ref) < 1e-10


@pytest.mark.parametrize("precision,tol", [(B.FP64, 1e-12), (B.FP32, 1e-5)])
@pytest.mark.parametrize("e", [4, 6, 10, 16])
def test_anterpolation_by_clusters_and_by_blocks(e, precision, tol):
    """A problem of 4^3 blocks has 8 or 27 receiving blocks per coarse level, eight CTAs for each; sixteen of them in a
    batch have more than 120, one CTA for each."""
    prob = dict(bd_base=(-4 * e,) * 3, bd_extent=(8 * e,) * 3, blocks=[((-2 * e,) * 3, (4 * e,) * 3)])
    one = B.Solver(prob["bd_base"], prob["bd_extent"], e, 0.5, prob["blocks"], precision=precision)
    many = B.BatchSolver(e, 0.5, [prob] * 16, precision=precision)
    one.mac_variant(0)
    many.mac_variant(0)
    src = np.random.default_rng(e).standard_normal((many.n, e + 2, e + 2, e + 2))
    fs, ft = many.field(src), many.field()
    many.apply_lgf(fs, ft)
    out, a, b = many.split(many.download(ft)), one.field(), one.field()
    for i in (0, 15):
        one.upload(a, many.split(src)[i])
        one.apply_lgf(a, b)
        assert rel_linf(out[i], one.download(b)) < tol


@pytest.mark.parametrize("n", [1, 7, 8, 33])
def test_ib_few_points(n):
    """Point counts around a CTA's eight points of the projection; 1e-9 as for the whole sphere's force solve."""
    case = S.SphereIB("small")
    args = (case.bd_base, case.bd_extent, case.block_extent, case.dx_base, case.blocks)
    o = O.Domain(*args, n_levels=case.n_levels, predicate=case.predicate)
    g = B.Solver(*args, n_levels=case.n_levels, predicate=case.predicate)
    X = O.sphere_points(case.dx_base, o.depth - 1 - o.base_level, case.ibph)[:n]
    u = case.velocity(o)
    f_ref, _, _ = o.ib_solve(X, case.Re, u, 7e-4, 1e-3, 40)
    g.ib_set_points(X, case.Re)
    f, _ = g.ib_solve([g.field(u[k]) for k in range(3)], 7e-4, 1e-3, 40)
    assert rel_linf(f, f_ref) < 1e-9
