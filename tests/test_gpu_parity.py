"""GPU parity: every CUDA path against the CPU oracle on the same seeded inputs,
through the C ABI (chidg_b200.api wraps include/chidg_gpu.h).

Tolerances (FP64 mode): matvec and ILU sweeps 1e-12 relative to the vector
norm (summation order differs from the oracle); factor blocks 1e-10 relative
to the block norm (pivoted inverses of 135 x 135 blocks); FGMRES: same
iteration count, residual history within 1e-8 relative, solution within
1e-10 relative.
"""
import numpy as np
import pytest

from chidg_b200 import _lib, api, mesh
from oracle import oracle as O
from tests import kat_util

pytestmark = pytest.mark.gpu


def relerr(a, b):
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


def setup(shape, P, nt=1, sub=(1, 1, 1), seed=1, nvars=5):
    pat = mesh.box_pattern(*shape, nvars, mesh.nterms_of_order(P), ntime=nt, subdomains=sub)
    vals = mesh.synth_values(pat, seed=seed)
    Ao = O.OracleMatrix(pat)
    Ao.set_values(vals)
    Ag = api.ChidgMatrix(pat)
    Ag.upload(vals)
    return pat, vals, Ao, Ag


CASES = [((4, 3, 2), 1, 1), ((3, 3, 3), 2, 1), ((2, 2, 2), 1, 3), ((5, 1, 1), 0, 1)]


@pytest.mark.parametrize("shape,P,nt", CASES)
def test_matvec(shape, P, nt):
    pat, vals, Ao, Ag = setup(shape, P, nt)
    x = mesh.synth_vector(Ao.n, seed=2)
    y = api.chidg_mv(Ag, api.ChidgVector(Ag, x)).download()
    assert relerr(y, Ao.mv(x)) < 1e-13


def test_dot_norm_axpy():
    pat, vals, Ao, Ag = setup((3, 3, 3), 1)
    x = mesh.synth_vector(Ao.n, seed=3)
    y = mesh.synth_vector(Ao.n, seed=4)
    xg, yg = api.ChidgVector(Ag, x), api.ChidgVector(Ag, y)
    assert api.dot(xg, yg) == pytest.approx(float(x @ y), rel=1e-13)
    assert xg.norm() == pytest.approx(float(np.linalg.norm(x)), rel=1e-13)
    yg.axpy(-0.5, xg)
    assert relerr(yg.download(), y - 0.5 * x) < 1e-15


@pytest.mark.parametrize("schedule", ["levels", "dataflow", "tasks", "stream"])
@pytest.mark.parametrize("kind", ["ilu0", "jacobi"])
@pytest.mark.parametrize("shape,P,nt", CASES)
def test_precon_factor_and_apply(kind, shape, P, nt, schedule):
    pat, vals, Ao, Ag = setup(shape, P, nt, seed=5)
    Mo = O.OraclePrecon(Ao, kind)
    Mo.update()
    Mg = api.create_preconditioner(kind, schedule=schedule)
    Mg.update(Ag)
    LDo, LDg = Mo.LD(), Mg.LD()
    voff, _ = pat.value_offsets()
    nr, nc = pat.block_dims()
    worst = 0.0
    for k in range(pat.nblocks):
        a = LDo[voff[k]:voff[k] + nr[k] * nc[k]]
        if not np.any(a):
            continue
        worst = max(worst, relerr(LDg[voff[k]:voff[k] + nr[k] * nc[k]], a))
    assert worst < 1e-10
    v = mesh.synth_vector(Ao.n, seed=6)
    z = Mg.apply(Ag, api.ChidgVector(Ag, v)).download()
    assert relerr(z, Mo.apply(v)) < 1e-11


@pytest.mark.parametrize("schedule", ["levels", "dataflow", "tasks", "stream"])
@pytest.mark.parametrize("shape,P,sub", [((4, 4, 2), 1, (2, 2, 1)), ((4, 4, 4), 0, (2, 2, 2)), ((6, 3, 3), 1, (3, 1, 1))])
def test_rasilu0(shape, P, sub, schedule):
    pat, vals, Ao, Ag = setup(shape, P, 1, sub=sub, seed=7)
    Mo = O.OraclePrecon(Ao, "rasilu0")
    Mo.update()
    Mg = api.create_preconditioner("rasilu0", schedule=schedule)
    Mg.update(Ag)
    v = mesh.synth_vector(Ao.n, seed=8)
    z = Mg.apply(Ag, api.ChidgVector(Ag, v)).download()
    assert relerr(z, Mo.apply(v)) < 1e-11


@pytest.mark.parametrize("prec,shape,P,nt,orth", [("ilu0", (4, 3, 3), 1, 1, "CGS"), ("ilu0", (3, 3, 3), 2, 1, "CGS"),
                                                  ("ilu0", (3, 3, 2), 1, 1, "MGS"), ("jacobi", (3, 3, 3), 1, 1, "CGS"),
                                                  ("ilu0", (2, 2, 2), 1, 3, "CGS"), ("rasilu0", (4, 4, 2), 1, 1, "CGS")])
def test_fgmres_parity(prec, shape, P, nt, orth):
    sub = (2, 2, 1) if prec == "rasilu0" else (1, 1, 1)
    pat, vals, Ao, Ag = setup(shape, P, nt, sub=sub, seed=9)
    b = mesh.synth_vector(Ao.n, seed=10)
    opts = dict(tol=0.0, rtol=1e-8, nkrylov=12, inner_fgmres=0, nmax=400, orthogonalization=orth)
    xo, ro = O.fgmres(Ao, O.OraclePrecon(Ao, prec), b, O.default_opts(**opts))
    solver = api.create_linear_solver("fgmres", **opts)
    xg = api.ChidgVector(Ag)
    solver.solve(Ag, xg, api.ChidgVector(Ag, b), api.create_preconditioner(prec))
    assert solver.niter == ro["niter"]
    assert relerr(solver.hist, ro["hist"]) < 1e-8
    assert relerr(xg.download(), xo) < 1e-10
    assert solver.residual_norm == pytest.approx(ro["residual_norm"], rel=1e-6)


@pytest.mark.parametrize("kind,sub", [("ilu0", (1, 1, 1)), ("rasilu0", (2, 2, 2))])
def test_schedules_bitwise_identical(kind, sub):
    """Both sweep schedules run the same per-row arithmetic."""
    pat, vals, Ao, Ag = setup((6, 6, 4), 1, sub=sub, seed=22)
    v = api.ChidgVector(Ag, mesh.synth_vector(Ao.n, seed=23))
    out = []
    for sched in ("levels", "dataflow"):
        M = api.create_preconditioner(kind, schedule=sched)
        M.update(Ag)
        out.append(M.apply(Ag, v).download())
    assert np.array_equal(out[0], out[1])


@pytest.mark.parametrize("shape,P", [((2, 2, 2), 3), ((3, 2, 2), 4), ((7, 7, 7), 1)])
def test_stream_sweeps_block_sizes(shape, P):
    """Streamed sweeps with 320- and 625-row blocks (several rows per consumer
    thread, several column chunks per block) and with 343 small-block rows."""
    pat, vals, Ao, Ag = setup(shape, P, seed=24)
    Mo = O.OraclePrecon(Ao, "ilu0")
    Mo.update()
    Mg = api.create_preconditioner("ilu0", schedule="stream")
    Mg.update(Ag)
    v = mesh.synth_vector(Ao.n, seed=25)
    z = Mg.apply(Ag, api.ChidgVector(Ag, v)).download()
    assert relerr(z, Mo.apply(v)) < 1e-11


def test_stream_sweeps_deterministic():
    """The streamed sweeps' sums have a fixed order whichever CTA runs a task."""
    pat, vals, Ao, Ag = setup((6, 6, 4), 2, seed=26)
    v = api.ChidgVector(Ag, mesh.synth_vector(Ao.n, seed=27))
    M = api.create_preconditioner("ilu0", schedule="stream")
    M.update(Ag)
    z1 = M.apply(Ag, v).download()
    z2 = M.apply(Ag, v).download()
    assert np.array_equal(z1, z2)
    M.set_schedule("tasks")
    assert relerr(M.apply(Ag, v).download(), z1) < 1e-13


@pytest.mark.parametrize("precision,P", [("mixed_fp32", 2), ("mixed_bf16", 2), ("mixed_precon_fp32", 2),
                                         ("mixed_fp32", 3), ("mixed_bf16", 3)])
def test_stream_sweeps_mixed_precision(precision, P):
    """Every mixed mode reaches the FP64 residual target; with P3 (320-row
    blocks) the FP32 factorisation takes the large blocks' products on the
    FP32 SIMT kernel."""
    pat, vals, Ao, Ag = setup((4, 4, 4) if P == 2 else (3, 2, 2), P, seed=28)
    b = mesh.synth_vector(Ao.n, seed=29)
    solver = api.create_linear_solver("fgmres", tol=0.0, rtol=1e-8, nkrylov=10, inner_fgmres=0, nmax=50,
                                      precision=precision, mixed_inner_nkrylov=20, mixed_inner_rtol=1e-2,
                                      mixed_inner_nmax=40)
    xg = api.ChidgVector(Ag)
    solver.solve(Ag, xg, api.ChidgVector(Ag, b), api.create_preconditioner("ilu0", schedule="stream"))
    assert solver.residual_norm <= 1.5e-8 * solver.r0norm_initial
    r = b - Ao.mv(xg.download())
    assert np.linalg.norm(r) <= 2e-8 * np.linalg.norm(b)


@pytest.mark.parametrize("nvars,P", [(3, 2), (4, 2), (1, 4), (2, 3), (5, 2)])
def test_factor_inverse_sizes_one_cta(nvars, P):
    """Diagonal inverses of 81..136-row blocks (panels of eight columns and
    tensor-core updates by one CTA, partial tiles included) against the oracle's
    DGETRF/DGETRI."""
    pat, vals, Ao, Ag = setup((3, 2, 2), P, seed=30, nvars=nvars)
    Mo = O.OraclePrecon(Ao, "ilu0")
    Mo.update()
    Mg = api.create_preconditioner("ilu0")
    Mg.update(Ag)
    LDo, LDg = Mo.LD(), Mg.LD()
    voff, _ = pat.value_offsets()
    nr, nc = pat.block_dims()
    worst = 0.0
    for k in range(pat.nblocks):
        a = LDo[voff[k]:voff[k] + nr[k] * nc[k]]
        if np.any(a):
            worst = max(worst, relerr(LDg[voff[k]:voff[k] + nr[k] * nc[k]], a))
    assert worst < 1e-10


@pytest.mark.parametrize("nvars", [3, 4, 5])
def test_factor_inverse_sizes_clusters(nvars):
    """Diagonal inverses of 192..320-row blocks (P3; the same panels, by clusters
    of two to five CTAs) and the L blocks built from them, against the oracle's
    DGETRF/DGETRI and ILU0."""
    pat, vals, Ao, Ag = setup((2, 2, 1), 3, seed=36, nvars=nvars)
    Mo = O.OraclePrecon(Ao, "ilu0")
    Mo.update()
    Mg = api.create_preconditioner("ilu0")
    Mg.update(Ag)
    LDo, LDg = Mo.LD(), Mg.LD()
    voff, _ = pat.value_offsets()
    nr, nc = pat.block_dims()
    worst = 0.0
    for k in range(pat.nblocks):
        a = LDo[voff[k]:voff[k] + nr[k] * nc[k]]
        if np.any(a):
            worst = max(worst, relerr(LDg[voff[k]:voff[k] + nr[k] * nc[k]], a))
    assert worst < 1e-10


@pytest.mark.parametrize("P", [2, 3])
def test_inverse_with_row_permuted_blocks(P):
    """Diagonal blocks whose rows are shuffled, so that partial pivoting takes
    off-diagonal pivots and the inverse kernels undo a long permutation
    (135 rows: one CTA; 320 rows: a cluster of five), against
    the oracle's DGETRF/DGETRI (block Jacobi: the inverses alone)."""
    pat, vals, Ao, Ag = setup((2, 2, 1), P, seed=38)
    voff, _ = pat.value_offsets()
    nr, nc = pat.block_dims()
    rng = np.random.default_rng(39)
    bad = vals.copy()
    for k in range(pat.nblocks):
        if pat.blk_row_elem[k] == pat.blk_col_elem[k]:
            blk = bad[voff[k]:voff[k] + nr[k] * nc[k]].reshape(nc[k], nr[k])   # [column][row]
            blk[:, :] = blk[:, rng.permutation(nr[k])]
    Ao.set_values(bad)
    Ag.upload(bad)
    Mo = O.OraclePrecon(Ao, "jacobi")
    Mo.update()
    Mg = api.create_preconditioner("jacobi")
    Mg.update(Ag)
    LDo, LDg = Mo.LD(), Mg.LD()
    worst = 0.0
    for k in range(pat.nblocks):
        a = LDo[voff[k]:voff[k] + nr[k] * nc[k]]
        if np.any(a):
            worst = max(worst, relerr(LDg[voff[k]:voff[k] + nr[k] * nc[k]], a))
    assert worst < 1e-10


def test_singular_block_reports_element_cluster_inverse():
    pat, vals, Ao, Ag = setup((2, 2, 1), 3, seed=37)
    voff, _ = pat.value_offsets()
    nr, nc = pat.block_dims()
    k = int(np.nonzero((pat.blk_row_elem == 2) & (pat.blk_col_elem == 2))[0][0])
    bad = vals.copy()
    blk = bad[voff[k]:voff[k] + nr[k] * nc[k]].reshape(nc[k], nr[k])
    blk[:, 5] = 0.0                     # a zero row: singular
    Ag.upload(bad)
    M = api.create_preconditioner("jacobi")
    with pytest.raises(_lib.ChidgGpuError) as ei:
        M.update(Ag)
    assert ei.value.code == _lib.ESINGULAR and ei.value.element == 2


def test_singular_block_reports_element_one_cta_inverse():
    pat, vals, Ao, Ag = setup((3, 2, 2), 2, seed=31)
    voff, _ = pat.value_offsets()
    nr, nc = pat.block_dims()
    k = int(np.nonzero((pat.blk_row_elem == 7) & (pat.blk_col_elem == 7))[0][0])
    bad = vals.copy()
    blk = bad[voff[k]:voff[k] + nr[k] * nc[k]].reshape(nc[k], nr[k])
    blk[:, 3] = 0.0                     # a zero row: singular
    Ag.upload(bad)
    M = api.create_preconditioner("jacobi")
    with pytest.raises(_lib.ChidgGpuError) as ei:
        M.update(Ag)
    assert ei.value.code == _lib.ESINGULAR and ei.value.element == 7


@pytest.mark.parametrize("schedule", ["stream", "tasks"])
def test_precon_fp32_factors_close_to_fp64(schedule):
    """FP64 vectors through FP32 factors: the apply differs from the FP64 one by
    the rounding of the blocks (about 1e-7 relative), not more."""
    pat, vals, Ao, Ag = setup((4, 3, 3), 2, seed=32)
    v = api.ChidgVector(Ag, mesh.synth_vector(Ao.n, seed=33))
    M = api.create_preconditioner("ilu0", schedule=schedule)
    M.update(Ag)
    z64 = M.apply(Ag, v).download()
    M.update(Ag, precision="mixed_precon_fp32")
    assert relerr(M.apply(Ag, v).download(), z64) < 1e-12     # the plain apply stays FP64
    solver = api.create_linear_solver("fgmres", tol=0.0, rtol=1e-10, nkrylov=20, inner_fgmres=0, nmax=200,
                                      precision="mixed_precon_fp32")
    x = api.ChidgVector(Ag)
    b = mesh.synth_vector(Ao.n, seed=34)
    solver.solve(Ag, x, api.ChidgVector(Ag, b), M)
    xo, ro = O.fgmres(Ao, O.OraclePrecon(Ao, "ilu0"), b, O.default_opts(tol=0.0, rtol=1e-10, nkrylov=20,
                                                                        inner_fgmres=0, nmax=200))
    assert relerr(x.download(), xo) < 1e-8
    assert abs(solver.niter - ro["niter"]) <= 1


def test_precon_fp32_mode_uses_fp32_blocks():
    """After one FGMRES iteration the FP32-preconditioner iterate differs from
    the FP64 one by the rounding of the blocks: visible, and small."""
    pat, vals, Ao, Ag = setup((4, 3, 3), 2, seed=35)
    b = api.ChidgVector(Ag, mesh.synth_vector(Ao.n, seed=36))
    out = {}
    for prec in ("fp64", "mixed_precon_fp32"):
        solver = api.create_linear_solver("fgmres", tol=0.0, rtol=1e-14, nkrylov=1, inner_fgmres=0, nmax=1,
                                          precision=prec)
        x = api.ChidgVector(Ag)
        try:
            solver.solve(Ag, x, b, api.create_preconditioner("ilu0"))
        except _lib.ChidgGpuError as e:
            assert e.code == _lib.ENOTCONVERGED
        out[prec] = x.download()
    d = relerr(out["mixed_precon_fp32"], out["fp64"])
    assert 1e-12 < d < 1e-5, d


def test_upload_in_parts_matches_whole_upload():
    pat, vals, Ao, Ag = setup((3, 2, 2), 1, seed=37)
    whole = Ag.download()
    A2 = api.ChidgMatrix(pat)
    cut = [0, 5, len(vals) // 3, len(vals) // 3 + 1, len(vals)]
    A2.upload_parts([vals[a:b] for a, b in zip(cut[:-1], cut[1:])])
    assert np.array_equal(A2.download(), whole)
    v = mesh.synth_vector(Ao.n, seed=38)
    x = api.ChidgVector(A2)
    x.upload_parts([v[:7], v[7:]])
    assert np.array_equal(x.download(), v)
    with pytest.raises(_lib.ChidgGpuError) as ei:
        Ag.ctx.check(Ag.ctx.L.chidg_gpu_matrix_upload_range(A2.h, vals.ctypes.data, len(vals) - 3, 4), "range")
    assert ei.value.code == _lib.EINVAL


def test_fp32_factorisation_guards_the_fp64_apply():
    """MIXED_FP32 computes only FP32 factors: the FP64 apply and the factor
    download refuse until the next FP64 update, which then matches the oracle."""
    pat, vals, Ao, Ag = setup((3, 3, 2), 2, seed=39)
    M = api.create_preconditioner("ilu0")
    M.update(Ag, precision="mixed_fp32")
    v = api.ChidgVector(Ag, mesh.synth_vector(Ao.n, seed=40))
    with pytest.raises(_lib.ChidgGpuError) as ei:
        M.apply(Ag, v)
    assert ei.value.code == _lib.ESTATE
    M.update(Ag)
    Mo = O.OraclePrecon(Ao, "ilu0")
    Mo.update()
    assert relerr(M.apply(Ag, v).download(), Mo.apply(v.download())) < 1e-11


def test_fgmres_inner_default_options():
    """Reference defaults: inner FGMRES on, no controller (M refreshed per call)."""
    pat, vals, Ao, Ag = setup((3, 3, 2), 1, 1, seed=11)
    b = mesh.synth_vector(Ao.n, seed=12)
    opts = dict(tol=1e-9, rtol=1e-10, nkrylov=20, nmax=200)
    xo, ro = O.fgmres(Ao, O.OraclePrecon(Ao, "ilu0"), b, O.default_opts(**opts))
    solver = api.create_linear_solver("fgmres", **opts)
    xg = api.ChidgVector(Ag)
    solver.solve(Ag, xg, api.ChidgVector(Ag, b), api.create_preconditioner("ilu0"))
    assert solver.niter == ro["niter"]
    assert relerr(solver.hist, ro["hist"]) < 1e-8
    assert relerr(xg.download(), xo) < 1e-10


@pytest.mark.parametrize("name", ["ilu0", "ilu0_hb", "fgmres", "fgmres_ref"])
def test_reference_kats_on_gpu(name):
    case = kat_util.load_cases()[name]
    pat, vals, b = kat_util.build(case)
    A = api.ChidgMatrix(pat)
    A.upload(vals)
    eo = pat.elem_offsets()
    if name.startswith("ilu0"):
        M = api.create_preconditioner("ilu0")
        M.update(A)
        LD = M.LD()
        z = M.apply(A, api.ChidgVector(A, b)).download()
        for kind, idx, expect in case["asserts"]:
            if kind == "LD":
                assert LD[kat_util.ld_index(pat, *idx)] == pytest.approx(expect, rel=1e-15)
            else:
                e, i = idx
                assert abs(z[eo[e - 1] + i - 1] - expect) <= case["tol"]
    else:
        solver = api.create_linear_solver("fgmres", tol=case["solver_tol"], nmax=1000)
        x = api.ChidgVector(A)
        solver.solve(A, x, api.ChidgVector(A, b), api.create_preconditioner("identity"))
        xv = x.download()
        for kind, (e, i), expect in case["asserts"]:
            assert abs(xv[eo[e - 1] + i - 1] - expect) <= case["tol"]


@pytest.mark.parametrize("precision,kind", [("mixed_fp32", "ilu0"), ("mixed_bf16", "ilu0"),
                                            ("mixed_precon_fp32", "ilu0"), ("mixed_fp32", "rasilu0"),
                                            ("mixed_bf16", "rasilu0")])
def test_mixed_precision_reaches_fp64_accuracy(precision, kind):
    """Every mixed mode, with ILU0 and with RAS+ILU0 (2 x 2 x 2 subdomains,
    FP32 factorisation of the overlap rows), reaches the FP64 residual."""
    sub = (2, 2, 2) if kind == "rasilu0" else (1, 1, 1)
    pat, vals, Ao, Ag = setup((4, 4, 4), 1, sub=sub, seed=13)
    b = mesh.synth_vector(Ao.n, seed=14)
    xo, ro = O.fgmres(Ao, O.OraclePrecon(Ao, "ilu0"), b,
                      O.default_opts(tol=0.0, rtol=1e-12, nkrylov=40, inner_fgmres=0, nmax=400))
    solver = api.create_linear_solver("fgmres", tol=0.0, rtol=1e-8, nkrylov=10, inner_fgmres=0, nmax=50,
                                      precision=precision, mixed_inner_nkrylov=20, mixed_inner_rtol=1e-2,
                                      mixed_inner_nmax=40)
    xg = api.ChidgVector(Ag)
    solver.solve(Ag, xg, api.ChidgVector(Ag, b), api.create_preconditioner(kind))
    assert solver.residual_norm <= 1.5e-8 * solver.r0norm_initial
    assert relerr(xg.download(), xo) < 1e-6


def test_singular_block_reports_element():
    pat, vals, Ao, Ag = setup((3, 2, 2), 1, seed=15)
    voff, _ = pat.value_offsets()
    nr, nc = pat.block_dims()
    k = int(np.nonzero((pat.blk_row_elem == 4) & (pat.blk_col_elem == 4))[0][0])
    bad = vals.copy()
    bad[voff[k]:voff[k] + nr[k] * nc[k]] = 0.0
    Ag.upload(bad)
    M = api.create_preconditioner("jacobi")
    with pytest.raises(_lib.ChidgGpuError) as ei:
        M.update(Ag)
    assert ei.value.code == _lib.ESINGULAR and ei.value.element == 4


def test_nonfinite_rhs_reported():
    pat, vals, Ao, Ag = setup((3, 2, 2), 1, seed=16)
    b = mesh.synth_vector(Ao.n, seed=17)
    b[5] = np.nan
    solver = api.create_linear_solver("fgmres", tol=0.0, rtol=1e-8, nkrylov=10, inner_fgmres=0, nmax=20)
    with pytest.raises(_lib.ChidgGpuError) as ei:
        solver.solve(Ag, api.ChidgVector(Ag), api.ChidgVector(Ag, b), api.create_preconditioner("ilu0"))
    assert ei.value.code == _lib.ENONFINITE


def test_controller_reuses_factorisation():
    pat, vals, Ao, Ag = setup((3, 3, 2), 1, seed=18)
    b = api.ChidgVector(Ag, mesh.synth_vector(Ao.n, seed=19))
    M = api.create_preconditioner("ilu0")
    solver = api.create_linear_solver("fgmres", tol=0.0, rtol=1e-8, nkrylov=20, inner_fgmres=0, nmax=100,
                                      use_controller=True)
    x = api.ChidgVector(Ag)
    solver.solve(Ag, x, b, M)
    s1 = M.stamp
    solver.solve(Ag, x, b, M)
    assert M.stamp == s1 == Ag.stamp
    Ag.upload(vals * 1.0)     # a new assembly bumps the stamp -> refactor
    solver.solve(Ag, x, b, M)
    assert M.stamp == Ag.stamp and M.stamp != s1


def test_upload_blocks_equals_packed():
    pat, vals, Ao, Ag = setup((3, 2, 2), 1, seed=20)
    voff, _ = pat.value_offsets()
    nr, nc = pat.block_dims()
    blocks = [vals[voff[k]:voff[k] + nr[k] * nc[k]].reshape(nc[k], nr[k]).T for k in range(pat.nblocks)]
    A2 = api.ChidgMatrix(pat)
    A2.upload_blocks(blocks)
    assert np.array_equal(A2.download(), vals)


def test_scale_diagonal():
    pat, vals, Ao, Ag = setup((2, 2, 1), 1, seed=21)
    nt = int(pat.elem_nterms[0])
    nv = int(pat.elem_nvars[0])
    rng = np.random.default_rng(0)
    mass = rng.standard_normal((pat.nelem, nt, nt))
    scale = rng.standard_normal((pat.nelem, nv))
    Ag.scale_diagonal(np.ascontiguousarray(mass.transpose(0, 2, 1)).ravel(), scale.ravel())
    got = Ag.download()
    voff, _ = pat.value_offsets()
    b = nt * nv
    for k in range(pat.nblocks):
        e = pat.blk_row_elem[k]
        blk = vals[voff[k]:voff[k] + b * b].reshape(b, b).T.copy()
        if pat.blk_col_elem[k] == e:
            for f in range(nv):
                blk[f * nt:(f + 1) * nt, f * nt:(f + 1) * nt] += scale[e, f] * mass[e]
        assert np.allclose(got[voff[k]:voff[k] + b * b].reshape(b, b).T, blk, rtol=1e-15, atol=1e-15)


@pytest.mark.parametrize("shape,P,nt", [((3, 2, 2), 1, 1), ((2, 2, 2), 2, 3)])
def test_norm_fields_and_operators(shape, P, nt):
    """chidg_vector%norm_fields (per-field L2 norms over elements, time levels
    and modes) and the overloaded + - * / against numpy."""
    pat, vals, Ao, Ag = setup(shape, P, nt=nt, seed=111)
    x = mesh.synth_vector(Ao.n, seed=112)
    y = mesh.synth_vector(Ao.n, seed=113)
    xv, yv = api.ChidgVector(Ag, x), api.ChidgVector(Ag, y)
    nv, nterms = int(pat.elem_nvars[0]), int(pat.elem_nterms[0])
    per = x.reshape(pat.nelem, nt, nv, nterms)
    expect = np.sqrt((per ** 2).sum(axis=(0, 1, 3)))
    assert np.allclose(xv.norm_fields(), expect, rtol=1e-13)
    assert np.allclose((xv + yv).download(), x + y, rtol=0, atol=0)
    assert np.allclose((xv - yv).download(), x - y, rtol=0, atol=0)
    assert np.allclose((2.5 * xv).download(), 2.5 * x, rtol=0, atol=0)
    assert np.allclose((xv / 4.0).download(), x * 0.25, rtol=0, atol=0)
    assert np.allclose((-xv).download(), -x, rtol=0, atol=0)
    with pytest.raises(_lib.ChidgGpuError):
        xv.norm_fields(nv + 1)
