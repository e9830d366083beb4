"""Gradient of the elliptic solve (semtex_b200.autograd.helmholtz_solve)
against central finite differences (h = 1e-6, agreement to 1e-6 relative)
and the exact adjoint identity w^T (A(f + e) - A(f)) = (A^T w)^T e, with
inhomogeneous Dirichlet and mixed (Robin) boundaries, in 2D and 3D."""
import numpy as np
import pytest

import semtex_b200 as S
from semtex_b200 import sessions
from semtex_b200.autograd import helmholtz_solve, solve_physical

pytestmark = pytest.mark.gpu


def _session(tmp_path, nz):
    p = sessions.rect_session(str(tmp_path / f"adj{nz}"), 4, 3,
                              tokens={"N_P": 6, "N_Z": nz, "BETA": 1.0, "LAMBDA2": 2.0, "TOL_REL": 1e-14},
                              periodic_x=True, bcs={"w": {"c": "<M> 1.5;0.2"}})
    txt = open(p).read()
    txt = txt.replace("<GROUPS NUMBER=1>", "<GROUPS NUMBER=2>\n\t2\tz\tclamp")
    bc = "0.3+0.1*cos(z)" if nz > 1 else "0.3"
    txt = txt.replace("<BCS NUMBER=1>", f"<BCS NUMBER=2>\n\t2\tz\t1\n\t\t<D>\tc = {bc}\t</D>")
    out = []
    for ln in txt.splitlines():
        parts = ln.split("\t")
        if len(parts) >= 4 and parts[3] == "1" and "<B>" in ln:
            ln = ln.replace("<B>\tw\t</B>", "<B>\tz\t</B>")
        out.append(ln)
    open(p, "w").write("\n".join(out) + "\n")
    return p


@pytest.mark.parametrize("nz", [1, 8])
def test_solve_gradient(tmp_path, nz):
    import torch
    p = _session(tmp_path, nz)
    ctx = S.Context(p)
    sysm = S.ModalMatrixSys(ctx, "c", 2.0)
    dev = "cuda:0"
    rng = np.random.default_rng(nz)
    shape = (ctx.nz, ctx.nel, ctx.np, ctx.np)
    f0 = torch.tensor(rng.uniform(-1, 1, shape), device=dev)
    w = torch.tensor(rng.uniform(-1, 1, shape), device=dev)
    f = f0.clone().requires_grad_(True)
    u = helmholtz_solve(f, sysm)
    (w * u).sum().backward()
    grad = f.grad.detach()
    L = lambda x: float((w * solve_physical(sysm, x)).sum())
    for k in range(3):
        e = torch.tensor(rng.uniform(-1, 1, shape), device=dev)
        ge = float((grad * e).sum())
        lin = float((w * (solve_physical(sysm, f0 + e) - solve_physical(sysm, f0))).sum())
        assert abs(lin - ge) <= 1e-11 * abs(ge), (lin, ge)
        h = 1e-6
        fd = (L(f0 + h * e) - L(f0 - h * e)) / (2 * h)
        assert abs(fd - ge) <= 1e-6 * abs(ge), (fd, ge)
    sysm.close()
    ctx.close()


@pytest.mark.parametrize("method", ["DIRECT", "MIXED", "JACPCG"])
def test_solve_on_the_callers_stream(tmp_path, method):
    """The solve is ordered with the caller's stream only: forcings made and
    results used on a side stream right away, two systems' solves in turn, a
    strided forcing; against the host-buffer solve (round-off; the iteration's
    tolerance of 1e-14 on systems of condition below 1e5)."""
    import torch
    p = sessions.helmholtz_session(str(tmp_path / "st"), 4, 6, nz=6, lambda2=50.0,
                                   extra={"TOL_REL": 1e-14, "STEP_MAX": 2000})
    ctx = S.Context(p)
    systems = [S.ModalMatrixSys(ctx, "c", lam, method=getattr(S, method)) for lam in (50.0, 80.0)]
    shape = (ctx.nz, ctx.nel, ctx.np, ctx.np)
    f = np.random.default_rng(7).uniform(-1, 1, (3,) + shape)
    ref = [[s.solve_host(2.0 * x) for x in f] for s in systems]
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        # the three forcings strided, each made on the stream just before its use
        d = torch.from_numpy(np.ascontiguousarray(np.moveaxis(f, 0, -1))).cuda()
        got = []
        for s in systems:
            for i in range(3):
                x = (2.0 * d[..., i]).requires_grad_(True)
                u = helmholtz_solve(x, s)
                (g,) = torch.autograd.grad(u, x, torch.ones_like(u))
                got.append((u.detach() * 1.0, g))
                del x, u
    side.synchronize()
    tol = 1e-9 if method == "JACPCG" else 1e-12
    for k, (u, g) in enumerate(got):
        r = ref[k // 3][k % 3]
        assert np.linalg.norm(u.cpu().numpy() - r) <= tol * np.linalg.norm(r), k
        r = got[3 * (k // 3)][1]  # the gradient of a sum does not depend on the forcing
        assert float((g - r).norm()) <= tol * float(r.norm()), k
    for s in systems:
        s.close()
    ctx.close()


def test_failed_solve_leaves_the_streams_ordered(tmp_path, monkeypatch):
    """A solve that fails after work was queued: the caller's stream, on which
    its forcing may then be freed, still comes after that work."""
    import torch
    ctx = S.Context(sessions.helmholtz_session(str(tmp_path / "fs"), 2, 5, nz=4))
    sysm = S.ModalMatrixSys(ctx, "c", 1.0)
    f = torch.zeros((ctx.nz, ctx.nel, ctx.np, ctx.np), dtype=torch.float64, device="cuda")
    helmholtz_solve(f, sysm)
    torch.cuda.synchronize()

    def fail(self, forcing, system):
        torch.cuda._sleep(200_000_000)  # a tenth of a second on the context stream
        raise S.StxError(1, "made up")

    monkeypatch.setattr(S.Field, "solve", fail)
    with pytest.raises(S.StxError):
        helmholtz_solve(f, sysm)
    torch.cuda.current_stream().synchronize()
    assert ctx.torch_stream().query()
    torch.cuda.synchronize()
    sysm.close()
    ctx.close()


def test_reserve(tmp_path):
    from semtex_b200._lib import check, lib
    ctx = S.Context(sessions.helmholtz_session(str(tmp_path / "rs"), 3, 5, nz=4))
    sysm = S.ModalMatrixSys(ctx, "c", 1.0)
    f = np.random.default_rng(0).uniform(-1, 1, (4, 9, 5, 5))
    ref = sysm.solve_host(f)
    for n in (1, 3, 2):
        check(lib().stx_modal_reserve(sysm.handle, n))
    got = sysm.solve_host(f)
    assert np.linalg.norm(got - ref) <= 1e-12 * np.linalg.norm(ref)
    for n in (0, 4):
        with pytest.raises(S.StxError):
            check(lib().stx_modal_reserve(sysm.handle, n))
    pcg = S.ModalMatrixSys(ctx, "c", 1.0, method=S.JACPCG)
    with pytest.raises(S.StxError):
        check(lib().stx_modal_reserve(pcg.handle, 1))
    pcg.close()
    sysm.close()
    ctx.close()
