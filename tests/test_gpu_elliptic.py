"""GPU parity of the condensed Helmholtz solve against the oracle (FP64).

Bar: relative L2 difference <= 1e-10 between the CUDA path (through the C
ABI) and the oracle's restatement of Field::solve on the same session and
forcing; plus agreement with the analytic solutions the sessions carry.
"""
import os

import numpy as np
import pytest

import semtex_oracle as O
import semtex_b200 as S
from semtex_b200 import sessions

from conftest import SESSIONS

pytestmark = pytest.mark.gpu
TOL = 1e-10


def rel_l2(a, b):
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


@pytest.mark.parametrize("name", ["helmholtz1", "poisson1", "laplace1", "laplace4", "laplace3", "mixed1"])
@pytest.mark.parametrize("iterative", [False, True])
def test_reference_sessions(name, iterative):
    path = os.path.join(SESSIONS, name)
    ov = {"ITERATIVE": 1, "TOL_REL": 1e-14} if iterative else None
    u = S.elliptic(path, overrides=ov, iterative=iterative)
    P, U = O.elliptic(path, ov)
    assert rel_l2(u, U) < (1e-9 if iterative else TOL)


def _random_case(tmp_path, n, np_, nz, seed, perturb=0.0):
    rng = np.random.default_rng(seed)
    xs = ys = None
    if perturb:
        xs = np.linspace(0, 1, n + 1)
        ys = np.linspace(0, 1, n + 1)
        xs[1:-1] += perturb * rng.uniform(-1, 1, n - 1) / n
        ys[1:-1] += perturb * rng.uniform(-1, 1, n - 1) / n
    p = sessions.helmholtz_session(str(tmp_path / f"r{seed}"), n, np_, nz=nz, lambda2=1.0, beta=1.0,
                                   xs=xs, ys=ys)
    ctx = S.Context(p)
    x, y = ctx.mesh_coords()
    f = rng.uniform(-1, 1, (nz, n * n, np_, np_))
    return p, ctx, f


@pytest.mark.parametrize("n,np_,nz,perturb", [(4, 6, 8, 0.0), (5, 7, 6, 0.3), (3, 11, 4, 0.0), (6, 5, 1, 0.25)])
def test_random_forcing_fourier(tmp_path, n, np_, nz, perturb):
    p, ctx, f = _random_case(tmp_path, n, np_, nz, seed=n * 100 + np_, perturb=perturb)
    sysm = S.ModalMatrixSys(ctx, "c", 1.0)
    u = sysm.solve_host(f)
    P, U = O.elliptic(p, forcing_phys=f)
    assert rel_l2(u, U) < TOL
    if perturb:
        assert ctx.families() > 1


def test_two_calls_in_a_row_identical(tmp_path):
    p, ctx, f = _random_case(tmp_path, 4, 6, 8, seed=7)
    sysm = S.ModalMatrixSys(ctx, "c", 1.0)
    u1 = sysm.solve_host(f).copy()
    u2 = sysm.solve_host(f)
    assert rel_l2(u1, u2) < 1e-14
    assert sysm.status() == 0   # every bounded wait met its copy


def test_device_solve_and_transform(tmp_path):
    import torch
    p, ctx, f = _random_case(tmp_path, 4, 6, 8, seed=11)
    F = ctx.new_field("f").load_physical(f)
    F.transform(S.FORWARD)
    fo = O.dft_forward(f)
    got = F.to_numpy()
    assert rel_l2(got, fo) < 1e-14
    F.zero_nyquist()
    U = ctx.new_field("c")
    sysm = S.ModalMatrixSys(ctx, "c", 1.0)
    U.solve(F, sysm)
    U.transform(S.INVERSE)
    P, Uo = O.elliptic(p, forcing_phys=f)
    assert rel_l2(U.to_numpy(), Uo) < TOL


@pytest.mark.parametrize("nz", [4, 6, 10, 12, 14, 64, 96])
def test_transform_roundtrip_odd_factors(tmp_path, nz):
    # radix 4/2/3/5 FFT paths, and the DFT for a factor outside 2, 3, 5 (14)
    p = sessions.helmholtz_session(str(tmp_path / "t"), 2, 5, nz=nz)
    ctx = S.Context(p)
    rng = np.random.default_rng(nz)
    f = rng.standard_normal((nz, 4, 5, 5))
    F = ctx.new_field().load_physical(f)
    F.transform(S.FORWARD)
    assert rel_l2(F.to_numpy(), O.dft_forward(f)) < 1e-14
    F.transform(S.INVERSE)
    assert rel_l2(F.to_numpy(), f) < 1e-14


@pytest.mark.parametrize("n,np_,nz,perturb", [(8, 9, 8, 0.0), (8, 7, 6, 0.3)])
def test_mixed_precision_refined(tmp_path, n, np_, nz, perturb):
    """STX_MIXED: FP32 skeleton matrices (FP64 sums) with FP64 iterative
    refinement on the skeleton system reaches the FP64 oracle to 1e-10 (the
    default two refinements); without refinement (STX_REFINE = 0) the FP32
    matrices alone leave an error above 1e-9, so the refinement does the work."""
    p, ctx, f = _random_case(tmp_path, n, np_, nz, seed=n * 10 + np_, perturb=perturb)
    plain = S.ModalMatrixSys(ctx, "c", 1.0).solve_host(f)
    mixed = S.ModalMatrixSys(ctx, "c", 1.0, method=S.MIXED).solve_host(f)
    P, U = O.elliptic(p, forcing_phys=f)
    assert rel_l2(plain, U) < TOL
    assert rel_l2(mixed, U) < TOL, rel_l2(mixed, U)
    ctx0 = S.Context(p, overrides={"STX_REFINE": 0})
    none = S.ModalMatrixSys(ctx0, "c", 1.0, method=S.MIXED).solve_host(f)
    assert rel_l2(none, U) > 1e-9, rel_l2(none, U)


def test_mixed_precision_rejects_singular_systems():
    ctx = S.Context(os.path.join(SESSIONS, "taylor2"))
    with pytest.raises(S.StxError):
        S.ModalMatrixSys(ctx, "p", 0.0, method=S.MIXED)


@pytest.mark.parametrize("nf", [3, 2])
def test_multi_field_solve_matches_single(tmp_path, nf):
    """stx_field_solve_multi: velocity systems that share their matrices are
    solved with one skeleton pass for all fields; the results equal the
    one-by-one solves (round-off) and the oracle (1e-10)."""
    p = sessions.channel_session(str(tmp_path / "mf"), 4, 3, 7, 8, extra={"TOL_REL": 1e-14})
    ctx = S.Context(p)
    lam = 3.7
    names = "uvw"[:nf]
    systems = [S.ModalMatrixSys(ctx, c, lam) for c in names]
    rng = np.random.default_rng(nf)
    fs, single, multi, phys = [], [], [], []
    for c in names:
        f = rng.uniform(-1, 1, (ctx.nz, ctx.nel, ctx.np, ctx.np))
        phys.append(f)
        fs.append(ctx.new_field("f" + c).load_physical(f).transform(S.FORWARD).zero_nyquist())
        single.append(ctx.new_field("s" + c))
        multi.append(ctx.new_field("m" + c))
    for sys_, F, U in zip(systems, fs, single):
        U.solve(F, sys_)
    S.solve_multi(systems, fs, multi)
    P = O.Problem(O.read_session(p))
    for i, c in enumerate(names):
        a, b = multi[i].to_numpy(), single[i].to_numpy()
        assert rel_l2(a, b) < 1e-13, (c, rel_l2(a, b))
        F = O.dft_forward(phys[i])
        F[1] = 0.0
        Uo = P.solve(c, F, np.zeros_like(F), P.modal_systems(c, lam), P.bc_lines(c))
        Uo[1] = 0.0
        assert rel_l2(a, Uo) < TOL, (c, rel_l2(a, Uo))
    for sys_ in systems:
        sys_.close()
    ctx.close()



def _robin_session(path, nx, ny, np_, nz, K, C):
    """Periodic in x, Dirichlet 0 at y = 0, mixed dc/dn + K (c - C) = 0 at y = 1."""
    p = sessions.rect_session(path, nx, ny, tokens={"N_P": np_, "N_Z": nz, "BETA": 1.0, "LAMBDA2": 1.0,
                                                     "TOL_REL": 1e-14},
                              periodic_x=True, bcs={"w": {"c": f"<M> {K};{C}"}})
    txt = open(p).read()
    txt = txt.replace("<GROUPS NUMBER=1>", "<GROUPS NUMBER=2>\n\t2\tz\tclamp")
    txt = txt.replace("<BCS NUMBER=1>", "<BCS NUMBER=2>\n\t2\tz\t1\n\t\t<D>\tc = 0\t</D>")
    out = []
    for ln in txt.splitlines():
        parts = ln.split("\t")
        if len(parts) >= 4 and parts[3] == "1" and "<B>" in ln:   # side 1: bottom
            ln = ln.replace("<B>\tw\t</B>", "<B>\tz\t</B>")
        out.append(ln)
    open(p, "w").write("\n".join(out) + "\n")
    return p


@pytest.mark.parametrize("solver", ["twolevel", "band", "pcg"])
def test_mixed_bc_fourier(tmp_path, solver):
    """Mixed (Robin) BCs (src/condition.cpp:295-435) in 3D, against the oracle:
    K C <1, w> on every plane, K <c, w> on the boundary-system diagonal."""
    p = _robin_session(str(tmp_path / "rb"), 8, 6, 7, 8, 2.5, 0.3)
    ov = {"STX_TWOLEVEL": 0} if solver == "band" else ({"ITERATIVE": 1} if solver == "pcg" else None)
    ctx = S.Context(p, ov)
    rng = np.random.default_rng(5)
    f = rng.uniform(-1, 1, (ctx.nz, ctx.nel, ctx.np, ctx.np))
    sysm = S.ModalMatrixSys(ctx, "c", 1.0, method=S.JACPCG if solver == "pcg" else S.DIRECT)
    u = sysm.solve_host(f)
    P, U = O.elliptic(p, {"ITERATIVE": 1} if solver == "pcg" else None, forcing_phys=f)
    assert rel_l2(u, U) < (1e-9 if solver == "pcg" else TOL), rel_l2(u, U)
    with pytest.raises(S.StxError):
        S.ModalMatrixSys(ctx, "c", 1.0, method=S.MIXED)
    sysm.close()
    ctx.close()


@pytest.mark.parametrize("n,np_,nz", [(4, 2, 4), (3, 3, 8), (5, 4, 2), (1, 5, 4), (2, 2, 1)])
def test_edge_sizes(tmp_path, n, np_, nz):
    """Linear elements (N_P = 2: no interior nodes), quadratics, N_Z = 2 (mean
    and Nyquist planes only), a single element; direct and PCG."""
    p, ctx, f = _random_case(tmp_path, n, np_, nz, seed=n * 1000 + np_ * 10 + nz)
    P, U = O.elliptic(p, forcing_phys=f)
    u = S.ModalMatrixSys(ctx, "c", 1.0).solve_host(f)
    assert rel_l2(u, U) < TOL, rel_l2(u, U)
    ctx2 = S.Context(p, {"ITERATIVE": 1, "TOL_REL": 1e-14})
    ui = S.ModalMatrixSys(ctx2, "c", 1.0, method=S.JACPCG).solve_host(f)
    assert rel_l2(ui, U) < 1e-9, rel_l2(ui, U)


# one instance of the iteration kernel each (N_P <= 4, 8, 12, 16 and above),
# one to sixteen blocks a plane, more elements than warps
@pytest.mark.parametrize("n,np_,nz", [(1, 4, 6), (3, 8, 4), (9, 9, 4), (10, 6, 22), (5, 12, 1), (2, 16, 8), (3, 18, 4)])
def test_pcg_sizes(tmp_path, n, np_, nz):
    """The iteration stops at a residual of 1e-14 of the right-hand side; the
    Jacobi-scaled condition number of these systems is below 1e5, so the
    solution is within 1e-9 of the oracle's."""
    rng = np.random.default_rng(n * 100 + np_)
    xs = np.linspace(0, 1, n + 1)
    xs[1:-1] += 0.2 * rng.uniform(-1, 1, n - 1) / n
    p = sessions.helmholtz_session(str(tmp_path / "pcg"), n, np_, nz=nz, lambda2=100.0, beta=1.0, xs=xs,
                                   extra={"TOL_REL": 1e-14, "STEP_MAX": 5000})
    ctx = S.Context(p)
    f = rng.uniform(-1, 1, (nz, n * n, np_, np_))
    u = S.ModalMatrixSys(ctx, "c", 100.0, method=S.JACPCG).solve_host(f)
    _, U = O.elliptic(p, forcing_phys=f)
    assert rel_l2(u, U) < 1e-9


def test_pcg_clusters_in_waves(tmp_path):
    """More clusters (47 planes of eight blocks) than are resident at once, so
    that blocks start while others of the grid are at work, solve after solve:
    every one within the iteration's tolerance (as above) of the oracle."""
    n, np_, nz = 8, 8, 48
    p = sessions.helmholtz_session(str(tmp_path / "pcgw"), n, np_, nz=nz, lambda2=100.0, beta=1.0,
                                   extra={"TOL_REL": 1e-14, "STEP_MAX": 5000})
    ctx = S.Context(p)
    f = np.random.default_rng(8).uniform(-1, 1, (nz, n * n, np_, np_))
    sysm = S.ModalMatrixSys(ctx, "c", 100.0, method=S.JACPCG)
    _, U = O.elliptic(p, forcing_phys=f)
    for _ in range(4):
        assert rel_l2(sysm.solve_host(f), U) < 1e-9
    sysm.close()
    ctx.close()


@pytest.mark.parametrize("n,np_,nz", [(1, 4, 6), (3, 8, 4), (9, 9, 4), (5, 12, 1), (2, 2, 2), (3, 18, 4)])
def test_pcg_by_launches(tmp_path, n, np_, nz):
    """The iteration as a chain of launches (STX_PCG_LAUNCHES = 1): the
    tolerance of test_pcg_sizes, and the iterations of the other form but for
    rounding in the last residuals."""
    p = sessions.helmholtz_session(str(tmp_path / "pcgl"), n, np_, nz=nz, lambda2=100.0, beta=1.0,
                                   extra={"TOL_REL": 1e-14, "STEP_MAX": 5000})
    f = np.random.default_rng(n * 10 + np_).uniform(-1, 1, (nz, n * n, np_, np_))
    _, U = O.elliptic(p, forcing_phys=f)
    its = []
    for form in (0, 1):
        ctx = S.Context(p, {"STX_PCG_LAUNCHES": form})
        sysm = S.ModalMatrixSys(ctx, "c", 100.0, method=S.JACPCG)
        assert rel_l2(sysm.solve_host(f), U) < 1e-9
        u = ctx.new_field("c").solve(ctx.new_field("f").load_physical(f), sysm)
        its.append(np.array(u.iterations))
        sysm.close()
        ctx.close()
    assert np.all(np.abs(its[0] - its[1]) <= 2 + its[0] // 10)


def test_pcg_of_a_large_plane(tmp_path):
    """One plane of many elements, which takes the launches by itself, against
    the direct solve (residual 1e-14, condition below 1e5)."""
    p = sessions.rect_session(str(tmp_path / "big"), 128, 32, tokens={"N_P": 7, "N_Z": 1, "TOL_REL": 1e-14,
                                                                      "STEP_MAX": 5000},
                              bcs={"w": {"c": "<D> 0.3*x"}})
    ctx = S.Context(p)
    f = np.random.default_rng(5).uniform(-1, 1, (1, ctx.nel, 7, 7))
    ref = S.ModalMatrixSys(ctx, "c", 1000.0).solve_host(f)
    assert rel_l2(S.ModalMatrixSys(ctx, "c", 1000.0, method=S.JACPCG).solve_host(f), ref) < 1e-9
    ctx.close()


# Patch products batched over a family's patches (STX_PATCH_GEMM = 1): one to
# six 8-column tiles a block and two column blocks, patch orders on both sides
# of the 32-row tiles and 64-row blocks, no interface at all, one plane
@pytest.mark.parametrize("nx,ny,np_,nz,cap,nf",
                         [(2, 2, 4, 1, 8, 1), (4, 2, 5, 4, 8, 3), (6, 4, 6, 6, 8, 3), (8, 8, 5, 4, 16, 3),
                          (8, 8, 9, 2, 16, 1), (12, 6, 7, 4, 36, 2), (16, 8, 4, 6, 8, 3), (5, 7, 8, 4, 16, 2)])
def test_patch_products_batched(tmp_path, nx, ny, np_, nz, cap, nf):
    p = sessions.channel_session(str(tmp_path / "pg"), nx, ny, np_, nz,
                                 extra={"TOL_REL": 1e-14, "STX_PATCH_CAP": cap, "STX_PATCH_GEMM": 1})
    ctx = S.Context(p)
    names = [c for c in "uvw" if c in ctx.fields][:nf]
    systems = [S.ModalMatrixSys(ctx, c, 2.3) for c in names]
    rng = np.random.default_rng(nx * 10 + np_)
    phys = [rng.uniform(-1, 1, (ctx.nz, ctx.nel, ctx.np, ctx.np)) for _ in names]
    fs = [ctx.new_field("f" + c).load_physical(f).transform(S.FORWARD).zero_nyquist() for c, f in zip(names, phys)]
    us = [ctx.new_field("u" + c) for c in names]
    S.solve_multi(systems, fs, us)
    P = O.Problem(O.read_session(p))
    for c, f, u in zip(names, phys, us):
        F = O.dft_forward(f)
        if nz > 1:
            F[1] = 0.0
        U = P.solve(c, F, np.zeros_like(F), P.modal_systems(c, 2.3), P.bc_lines(c))
        if nz > 1:
            U[1] = 0.0
        assert rel_l2(u.to_numpy(), U) < TOL, c
    for sys_ in systems:
        sys_.close()
    ctx.close()


# Blocks of the element kernels: parts of a chunk, row blocks (N_P >= 13), one
# or two planes of columns, one to ten rounds of nodes a lane; essential
# values that are not zero (the lift term) and a part smaller than the others
@pytest.mark.parametrize("nx,ny,np_,nz", [(1, 1, 3, 1), (9, 5, 4, 6), (6, 6, 9, 1), (7, 5, 10, 4), (5, 4, 11, 4),
                                          (4, 4, 13, 4), (3, 2, 16, 4), (3, 1, 17, 1)])
def test_element_block_shapes(tmp_path, nx, ny, np_, nz):
    p = sessions.rect_session(str(tmp_path / "eb"), nx, ny, tokens={"N_P": np_, "N_Z": nz, "LAMBDA2": 3.0, "BETA": 1.3},
                              bcs={"w": {"c": "<D> 1+x-2*y*y"}, "n": {"c": "<N> 0.5*x"}},
                              side_groups={"top": "n"})
    ctx = S.Context(p)
    f = np.random.default_rng(np_).uniform(-1, 1, (ctx.nz, ctx.nel, ctx.np, ctx.np))
    u = S.ModalMatrixSys(ctx, "c", 3.0).solve_host(f)
    _, U = O.elliptic(p, forcing_phys=f)
    assert rel_l2(u, U) < TOL


# A field solved in place: a recovery in one row block as it is (N_P = 9) or
# with larger blocks (12, 13), the chunk kernel (14..17) and the kernel of one
# element and plane a block (31)
@pytest.mark.parametrize("np_,nz,nf", [(2, 4, 1), (9, 4, 1), (12, 4, 1), (12, 4, 3), (13, 1, 1), (14, 6, 1), (16, 4, 3),
                                       (17, 1, 1), (31, 4, 1)])
def test_solve_in_place(tmp_path, np_, nz, nf):
    """The solution written over the forcing is the solution written elsewhere,
    up to the order of sums."""
    p = sessions.rect_session(str(tmp_path / "ip"), 3, 2, tokens={"N_P": np_, "N_Z": nz, "BETA": 1.3,
                                                                  "STX_MODE_GROUPS": 2},
                              bcs={"w": {"c": "<D> 1+x-2*y*y"}})
    ctx = S.Context(p)
    sysm = S.ModalMatrixSys(ctx, "c", 3.0)
    f = np.random.default_rng(np_).uniform(-1, 1, (nf, ctx.nz, ctx.nel, np_, np_))
    fs = [ctx.new_field("f").load_physical(x).zero_nyquist() for x in f]
    us = [ctx.new_field("c") for _ in fs]
    for F, U in zip(fs, us):
        U.solve(F, sysm)
    if nf == 1:
        fs[0].solve(fs[0], sysm)
    else:
        S.solve_multi([sysm] * nf, fs, fs)
    for F, U in zip(fs, us):
        a, b = F.to_numpy(), U.to_numpy()
        assert rel_l2(a, b) < 1e-12
    sysm.close()
    ctx.close()


# Essential values that are not zero, on elements with up to and more than 64
# boundary nodes, two-level and banded, natural and essential sides meeting
@pytest.mark.parametrize("nx,ny,np_,nz,two", [(5, 4, 2, 4, 1), (5, 4, 9, 6, 1), (5, 4, 9, 6, 0), (3, 2, 17, 4, 1),
                                              (2, 2, 18, 4, 1), (2, 1, 20, 1, 0)])
def test_essential_values(tmp_path, nx, ny, np_, nz, two):
    p = sessions.rect_session(str(tmp_path / "ess"), nx, ny,
                              tokens={"N_P": np_, "N_Z": nz, "LAMBDA2": 3.0, "BETA": 1.3, "STX_TWOLEVEL": two},
                              bcs={"w": {"c": "<D> 1+x-2*y*y"}, "n": {"c": "<N> 0.5*x"}, "m": {"c": "<D> sin(3*x)"}},
                              side_groups={"top": "n", "bottom": "m"})
    ctx = S.Context(p)
    f = np.random.default_rng(np_).uniform(-1, 1, (ctx.nz, ctx.nel, ctx.np, ctx.np))
    u = S.ModalMatrixSys(ctx, "c", 3.0).solve_host(f)
    _, U = O.elliptic(p, forcing_phys=f)
    assert rel_l2(u, U) < TOL
    ctx.close()


def test_patch_products_of_many_modes(tmp_path):
    """More (family, mode) groups than a grid has rows: the patch products are
    not batched over families, whatever the token says."""
    nz = 34000
    xs, ys = np.array([0.0, 0.2, 0.45, 0.75, 1.0]), np.array([0.0, 0.1, 0.25, 0.45, 0.6, 0.8, 1.0])
    p = sessions.rect_session(str(tmp_path / "pm"), 4, 6, xs=xs, ys=ys, tokens={"N_P": 3, "N_Z": nz, "BETA": 0.01,
                                                                         "STX_PATCH_CAP": 8},
                              periodic_x=True, periodic_y=True)
    assert S.patching(p, "c")["nfamily"] * (nz // 2) > 65535
    f = np.random.default_rng(1).uniform(-1, 1, (nz, 24, 3, 3))
    out = []
    for gemm in (0, 1):
        ctx = S.Context(p, {"STX_PATCH_GEMM": gemm})
        sysm = S.ModalMatrixSys(ctx, "c", 1.0)
        U = ctx.new_field("c").solve(ctx.new_field("f").load_physical(f).zero_nyquist(), sysm)
        out.append(U.to_numpy())
        sysm.close()
        ctx.close()
    assert rel_l2(out[1], out[0]) < 1e-13
