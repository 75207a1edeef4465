"""Factorisation and sweeps at the block sizes where their kernels change
shape: the factor products' tiles (8 x 8 accumulators, CTA tiles of at most 80
x 80), the inverses' panels of eight, row pairs of sixteen and cluster sizes (one
CTA up to 152 rows, two up to 208, three up to 256, four up to 288, five up to
320, six up to 352, seven up to 384, another kernel above), the sweeps' one-task
rows (up to 64) and column slices (three up to 160, eight above); matrices that
mix those sizes; and the sweeps' tasks where a level has blocks enough for a task
to take all slices of one."""
import numpy as np
import pytest

from chidg_b200 import _lib, api, mesh, tuning
from oracle import oracle as O

pytestmark = pytest.mark.gpu

# (fields, modes): block size is their product
SIZES = [(1, 1), (7, 1), (1, 8), (3, 3), (5, 8), (13, 5), (8, 10), (27, 3), (1, 127), (17, 8), (1, 137), (8, 19), (9, 17),
         (32, 5), (7, 23), (13, 16), (11, 19), (4, 64), (1, 257), (7, 40), (36, 8), (17, 17), (64, 5), (3, 107), (44, 8),
         (1, 353), (128, 3), (5, 77)]


def _relerr(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("nvars,nterms", SIZES, ids=[f"b{v * t}" for v, t in SIZES])
def test_factors_and_sweeps_by_block_size(nvars, nterms):
    pat = mesh.box_pattern(2, 2, 2 if nvars * nterms < 200 else 1, nvars, nterms)
    vals = mesh.synth_values(pat, seed=61)
    # rows of the diagonal blocks in another order: pivots off the diagonal
    rng = np.random.default_rng(62)
    voff, _ = pat.value_offsets()
    b = nvars * nterms
    for k in np.nonzero(np.asarray(pat.blk_face) == mesh.DIAG)[0][::2]:
        blk = vals[voff[k]:voff[k] + b * b].reshape(b, b)            # [column, row]
        blk[:] = blk[:, rng.permutation(b)]
    v = mesh.synth_vector(pat.vector_size(), seed=63)
    Ao = O.OracleMatrix(pat)
    Ao.set_values(vals)
    Ag = api.ChidgMatrix(pat)
    Ag.upload(vals)
    Mo, Mg = O.OraclePrecon(Ao, "ilu0"), api.create_preconditioner("ilu0")
    Mo.update()
    Mg.update(Ag)
    LDo, LDg = Mo.LD(), Mg.LD()
    # the permuted systems are worse conditioned: a bound relative to the block
    # inverses' condition, measured in FP64 by numpy
    dk = np.nonzero(np.asarray(pat.blk_face) == mesh.DIAG)[0]
    cond = max(np.linalg.cond(LDo[voff[k]:voff[k] + b * b].reshape(b, b)) for k in dk)
    tol = 64 * b * np.finfo(float).eps * max(1.0, cond)
    for k in range(pat.nblocks):
        o = LDo[voff[k]:voff[k] + b * b]
        if np.any(o):
            assert _relerr(LDg[voff[k]:voff[k] + b * b], o) < tol
    assert _relerr(Mg.apply(Ag, api.ChidgVector(Ag, v)).download(), Mo.apply(v)) < tol


@pytest.mark.parametrize("nvars,nterms", [(1, 1), (5, 8), (5, 27), (5, 64), (6, 64)], ids=["b1", "b40", "b135", "b320", "b384"])
def test_inverse_of_a_diagonal_block_is_the_correctly_rounded_quotient(nvars, nterms):
    """Pivots divide: a diagonal block's inverse holds 1 / d, bit for bit, over
    mantissas and the exponents of normal quotients and beyond (2^-1022 .. 2^1023)."""
    b = nvars * nterms
    pat = mesh.box_pattern(1 << 18 if b == 1 else 4, 1, 1, nvars, nterms)
    voff, nval = pat.value_offsets()
    diag = voff[np.asarray(pat.blk_face) == mesh.DIAG]
    rng = np.random.default_rng(64)
    d = np.ldexp(rng.uniform(1.0, 2.0, diag.size * b) * rng.choice([-1.0, 1.0], diag.size * b),
                 np.where(np.arange(diag.size * b) % 2, rng.integers(-1022, 1023, diag.size * b), 0))
    d = d.reshape(diag.size, b)
    vals = np.zeros(nval)
    at = diag[:, None] + (b + 1) * np.arange(b)
    vals[at] = d
    A = api.ChidgMatrix(pat)
    A.upload(vals)
    M = api.create_preconditioner("jacobi")
    M.update(A)
    want = np.zeros(nval)
    want[at] = 1.0 / d
    inside = (diag[:, None] + np.arange(b * b)).ravel()
    assert np.array_equal(M.LD()[inside], want[inside])


@pytest.mark.parametrize("sizes", [(216,), (257,), (320,), (352,), (209, 224, 243, 320), (321, 337, 352)],
                         ids=lambda s: "-".join(map(str, s)))
def test_inverses_of_many_large_blocks(sizes):
    """More blocks of 209 to 352 rows in one level than clusters fit the chip:
    one CTA a block.  Every second block's rows are shuffled; a singular one is
    reported by its element."""
    rng = np.random.default_rng(65)
    pat = mesh.box_pattern(120, 1, 1, 1, sizes[0])
    pat.elem_nterms[:] = rng.choice(sizes, pat.nelem)
    voff, nval = pat.value_offsets()
    diag = voff[np.asarray(pat.blk_face) == mesh.DIAG]
    vals = np.zeros(nval)
    blocks = []
    for k, (o, b) in enumerate(zip(diag, pat.elem_nterms)):
        D = np.eye(b) + 0.6 / np.sqrt(b) * rng.uniform(-1.0, 1.0, (b, b))
        blocks.append(D[rng.permutation(b)] if k % 2 else D)
        vals[o:o + b * b] = blocks[-1].ravel(order="F")
    A = api.ChidgMatrix(pat)
    A.upload(vals)
    M = api.create_preconditioner("jacobi")
    M.update(A)
    LD = M.LD()
    for o, D in zip(diag, blocks):
        b = len(D)
        # backward error of an inverse from LU with partial pivoting, times the condition
        tol = 64 * b * np.finfo(float).eps * np.linalg.cond(D)
        assert _relerr(LD[o:o + b * b].reshape(b, b).T, np.linalg.inv(D)) < tol
    b = int(pat.elem_nterms[77])
    vals[diag[77]:diag[77] + b * b].reshape(b, b)[:, 5] = 0.0              # a zero row
    A.upload(vals)
    with pytest.raises(_lib.ChidgGpuError) as ei:
        M.update(A)
    assert ei.value.code == _lib.ESINGULAR and ei.value.element == 77


@pytest.mark.parametrize("count", [3, 310])
@pytest.mark.parametrize("b", [64, 65, 160, 161, 256, 257, 385])
def test_jacobi_apply_by_block_size(b, count):
    """Slices of a programme without couplings: one task a row up to 64 rows,
    three slices up to 160 (grouped from 296 blocks on) and up to 256 (never
    grouped), eight above."""
    rng = np.random.default_rng(66)
    pat = mesh.box_pattern(count, 1, 1, 1, b)
    voff, nval = pat.value_offsets()
    diag = voff[np.asarray(pat.blk_face) == mesh.DIAG]
    D = np.eye(b) + 0.5 / np.sqrt(b) * rng.uniform(-1.0, 1.0, (count, b, b))
    vals = np.zeros(nval)
    for o, d in zip(diag, D):
        vals[o:o + b * b] = d.ravel(order="F")
    v = rng.uniform(-1.0, 1.0, (count, b))
    A = api.ChidgMatrix(pat)
    A.upload(vals)
    M = api.create_preconditioner("jacobi")
    M.update(A)
    z = M.apply(A, api.ChidgVector(A, v.ravel())).download().reshape(count, b)
    tol = 64 * b * np.finfo(float).eps * max(np.linalg.cond(d) for d in D)
    assert _relerr(z, np.linalg.solve(D, v[:, :, None])[:, :, 0]) < tol


def _mixed(pat, sizes, seed):
    """The pattern with one field and a block size from `sizes` per element, its
    values, and the oracle's and the library's matrices."""
    pat.elem_nterms[:] = np.random.default_rng(seed).choice(sizes, pat.nelem)
    vals = mesh.synth_values(pat, seed=seed)
    Ao, Ag = O.OracleMatrix(pat), api.ChidgMatrix(pat)
    Ao.set_values(vals)
    Ag.upload(vals)
    return vals, Ao, Ag


@pytest.mark.parametrize("sizes", [(40, 135, 320), (64, 65, 160, 161), (135, 320), (209, 243, 320), (321, 350, 384)],
                         ids=lambda s: "-".join(map(str, s)))
def test_mixed_block_sizes(sizes):
    """Rows of one, three and eight slices next to one another, and inverses of
    different sizes in one launch: factors, an application and a solve with the
    matvec rows in the backward sweep, against the oracle.  Tolerances as in
    test_gpu_edge.py."""
    pat = mesh.box_pattern(3, 3, 2, 1, sizes[0])
    vals, Ao, Ag = _mixed(pat, sizes, 71)
    Mo, Mg = O.OraclePrecon(Ao, "ilu0"), api.create_preconditioner("ilu0")
    Mo.update()
    Mg.update(Ag)
    voff, _ = pat.value_offsets()
    nr, nc = pat.block_dims()
    LDo, LDg = Mo.LD(), Mg.LD()
    for k in range(pat.nblocks):
        o = LDo[voff[k]:voff[k] + nr[k] * nc[k]]
        if np.any(o):
            assert _relerr(LDg[voff[k]:voff[k] + nr[k] * nc[k]], o) < 1e-10
    v = mesh.synth_vector(pat.vector_size(), seed=72)
    assert _relerr(Mg.apply(Ag, api.ChidgVector(Ag, v)).download(), Mo.apply(v)) < 1e-11
    opts = dict(tol=0.0, rtol=1e-8, nkrylov=20, inner_fgmres=0, nmax=400)
    xo, ro = O.fgmres(Ao, O.OraclePrecon(Ao, "ilu0"), v, O.default_opts(**opts))
    x, solver = api.ChidgVector(Ag), api.create_linear_solver("fgmres", **opts)
    solver.solve(Ag, x, api.ChidgVector(Ag, v), Mg)
    assert solver.niter == ro["niter"]
    assert _relerr(x.download(), xo) < 1e-10


def test_product_of_mixed_sizes_with_more_rows_than_ctas():
    """1716 rows of 5 and 40 equations: the rows by falling size, several turns of
    the CTAs."""
    pat = mesh.with_element_orders(mesh.box_pattern(11, 13, 12, 5, 8), np.random.default_rng(73).integers(0, 2, 1716))
    vals = mesh.synth_values(pat, seed=74)
    Ao, Ag = O.OracleMatrix(pat), api.ChidgMatrix(pat)
    Ao.set_values(vals)
    Ag.upload(vals)
    x = mesh.synth_vector(pat.vector_size(), seed=75)
    assert _relerr(api.chidg_mv(Ag, api.ChidgVector(Ag, x)).download(), Ao.mv(x)) < 1e-13


@pytest.mark.parametrize("b", [65, 161, 320])
def test_grouped_slices_give_the_sums_of_single_ones(b):
    """300 systems side by side: levels of 300 blocks, whose tasks take all slices of
    a block (three at 65 rows, eight above 160).  Bitwise the application of a
    system alone, whose tasks take a slice each; one of them against the oracle."""
    one = mesh.box_pattern(2, 1, 1, 1, b)
    union, sys_elem = mesh.concat_patterns([one] * 300)
    vals = np.concatenate([mesh.synth_values(one, seed=80 + s % 7) for s in range(300)])
    v = mesh.synth_vector(union.vector_size(), seed=81)
    A = api.ChidgMatrix(union)
    A.upload(vals)
    M = api.create_preconditioner("ilu0")
    M.update(A)
    z = M.apply(A, api.ChidgVector(A, v)).download().reshape(300, -1)
    v = v.reshape(300, -1)
    for s in (0, 1, 150, 299):
        A1 = api.ChidgMatrix(one)
        A1.upload(mesh.synth_values(one, seed=80 + s % 7))
        M1 = api.create_preconditioner("ilu0")
        M1.update(A1)
        assert np.array_equal(z[s], M1.apply(A1, api.ChidgVector(A1, v[s])).download())
    Ao = O.OracleMatrix(one)
    Ao.set_values(mesh.synth_values(one, seed=80))
    Mo = O.OraclePrecon(Ao, "ilu0")
    Mo.update()
    assert _relerr(z[0], Mo.apply(v[0])) < 1e-11


def test_rows_of_very_many_blocks():
    """One element with 240 time levels of 64 equations: the matvec rows of the
    backward sweep stage 15 360 columns, beside which four stages of the default
    ring do not fit.  Against the sweeps without matvec rows.  (A default that was
    read and set again is still a default.)"""
    for kind in range(4):
        tuning.set_shape(kind, 64, 8, tuning.get_shape(kind, 64, 8))
    pat = mesh.box_pattern(1, 1, 1, 8, 8, ntime=240)
    A = api.ChidgMatrix(pat)
    A.upload(mesh.synth_values(pat, seed=91))
    b = api.ChidgVector(A, mesh.synth_vector(pat.vector_size(), seed=92))
    xs = []
    for schedule in ("stream", "levels"):
        x = api.ChidgVector(A)
        solver = api.create_linear_solver("fgmres", tol=0.0, rtol=1e-30, nkrylov=4, nmax=4, inner_fgmres=0)
        solver.solve(A, x, b, api.create_preconditioner("ilu0", schedule=schedule))
        xs.append(x.download())
    assert _relerr(xs[0], xs[1]) < 1e-10


@pytest.mark.parametrize("nvars,nterms", [(5, 8), (7, 23), (5, 48), (5, 64)], ids=["b40", "b161", "b240", "b320"])
def test_subdomain_sweeps_by_block_size(nvars, nterms):
    """RASILU0 over eight subdomains (one task a row; two, three and four slices)
    against the oracle.  Tolerance as in test_gpu_edge.py."""
    pat = mesh.box_pattern(4, 2, 2, nvars, nterms, subdomains=(2, 2, 2))
    vals = mesh.synth_values(pat, seed=95)
    Ao, Ag = O.OracleMatrix(pat), api.ChidgMatrix(pat)
    Ao.set_values(vals)
    Ag.upload(vals)
    Mo, Mg = O.OraclePrecon(Ao, "rasilu0"), api.create_preconditioner("rasilu0")
    Mo.update()
    Mg.update(Ag)
    v = mesh.synth_vector(pat.vector_size(), seed=96)
    assert _relerr(Mg.apply(Ag, api.ChidgVector(Ag, v)).download(), Mo.apply(v)) < 1e-11
