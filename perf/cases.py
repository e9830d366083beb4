"""The work that programs have this library do, as cases that can be timed.

Three families, by their public entry points:

* elliptic solves (`Field.solve`, `ModalMatrixSys.solve_host`,
  `autograd.helmholtz_solve`, `Batch.launch`): one Helmholtz problem per
  Fourier mode on a rectangle of quads, Dirichlet walls;
* time stepping (`DNS.advance`): the Taylor--Green vortex and the plane
  channel, a run that is under way (each pass takes its next steps);
* gradients through time stepping (`autograd.dns_steps`).

A case is a dict of plain values; `kind` names the family member:

  solve   Field.solve, forcing and solution on the device in Fourier space
          (method "direct" | "mixed" | "pcg")
  host    ModalMatrixSys.solve_host: pinned physical forcing in, solution out
  grad    helmholtz_solve and its backward pass on device tensors
  batch   `count` uneven 2D problems replayed by one Batch.launch
  dns     DNS.advance(steps) of "channel" or "vortex"
  adjoint dns_steps forward and backward over `steps` steps

Sizes: nx x ny elements, np nodes per element side, nz Fourier planes.
"""

import ctypes
import math
import os
import tempfile

import numpy as np
import torch

import semtex_b200 as S
from semtex_b200 import _lib, autograd, sessions

# -- the cases ---------------------------------------------------------------


def listed():
    return [
        # the smallest call: one 2D problem of 4 x 4 elements (a steady 2D
        # Helmholtz run, or one scalar of a coupled code): launch latency
        dict(name="solve_2d_small", kind="solve", method="direct", nx=4, ny=4, np=9, nz=1, grading=0.0, lambda2=1.0),
        # a wall-graded mesh, every element of its own shape, an odd number
        # of elements: what most production meshes look like to the solver
        dict(name="solve_graded", kind="solve", method="direct", nx=9, ny=7, np=8, nz=20, grading=0.6, lambda2=10.0),
        # the batched 2D x Fourier solve of the benchmark
        dict(name="solve_headline", kind="solve", method="direct", nx=16, ny=16, np=11, nz=64, grading=0.0,
             lambda2=1.0),
        # the same problem with FP32 skeleton inverses and FP64 refinement
        dict(name="solve_mixed", kind="solve", method="mixed", nx=16, ny=16, np=11, nz=64, grading=0.0, lambda2=1.0),
        # the iterative option (`elliptic -i`, and the start-up steps of a DNS)
        dict(name="solve_pcg", kind="solve", method="pcg", nx=8, ny=8, np=9, nz=16, grading=0.0, lambda2=100.0),
        # a C++ caller's arrays in and out: PCIe copies and transforms included
        dict(name="solve_host", kind="host", nx=16, ny=16, np=11, nz=64, grading=0.0, lambda2=1.0),
        # the solve inside a torch graph: forward and backward
        dict(name="solve_grad", kind="grad", nx=12, ny=12, np=8, nz=32, grading=0.0, lambda2=1.0),
        # many independent problems of uneven size (4..32 elements a side,
        # order 6..12), one graph launch
        dict(name="batch_uneven", kind="batch", count=16, problems=20261203),
        # wall-bounded time stepping, high-order pressure BCs: small planes
        dict(name="dns_channel", kind="dns", flow="channel", nx=16, ny=8, np=9, nz=32, steps=42, dealias=0),
        # triply periodic time stepping, the largest state
        dict(name="dns_vortex", kind="dns", flow="vortex", nx=24, ny=24, np=9, nz=96, steps=42, dealias=0),
        # with 3/2-rule products, as under-resolved turbulence is run
        dict(name="dns_dealiased", kind="dns", flow="vortex", nx=16, ny=16, np=9, nz=64, steps=42, dealias=1),
        # gradient of a final state with respect to the initial one
        dict(name="dns_gradient", kind="adjoint", flow="channel", nx=12, ny=6, np=8, nz=24, steps=20, every=10,
             dealias=0),
    ]


# plane counts in use: products of 2, 3 and 5, and a few with a factor 7 or 11
_PLANES = (4, 6, 8, 10, 12, 14, 16, 18, 20, 22, 24, 28, 30, 32, 36, 40, 48, 54, 60, 64, 72, 80, 96)


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "mixed", "pcg", "host", "grad", "batch", "channel", "channel",
                       "vortex", "vortex", "adjoint"])
    if kind in ("solve", "mixed", "pcg", "host", "grad"):
        hi = 12 if kind == "pcg" else 24
        c = dict(kind=kind if kind in ("host", "grad") else "solve", nx=_log_int(rng, 3, hi), ny=_log_int(rng, 3, hi),
                 np=rng.randint(6, 13), nz=rng.choice((1,) + _PLANES) if kind != "pcg" else rng.choice((1, 4, 8, 16, 24)),
                 grading=rng.choice((0.0, 0.0, round(rng.uniform(0.2, 0.8), 3))),
                 lambda2=round(math.exp(rng.uniform(math.log(0.1), math.log(100.0))), 4))
        if kind in ("solve", "mixed", "pcg"):
            c["method"] = {"solve": "direct"}.get(kind, kind)
        if c["grading"]:  # every element its own matrices
            c["nx"], c["ny"], c["nz"] = min(c["nx"], 14), min(c["ny"], 14), min(c["nz"], 32)
        return c
    if kind == "batch":
        return dict(kind="batch", count=rng.randint(2, 20), problems=rng.randrange(1 << 30))
    if kind == "adjoint":
        return dict(kind="adjoint", flow="channel", nx=rng.randint(4, 12), ny=rng.randint(3, 6), np=rng.randint(5, 9),
                    nz=rng.choice((4, 8, 12, 16, 24)), steps=rng.randint(4, 20), every=rng.randint(3, 10), dealias=0)
    c = dict(kind="dns", flow=kind, nx=_log_int(rng, 4, 20), ny=_log_int(rng, 4, 20), np=rng.randint(5, 10),
             nz=rng.choice((1,) + _PLANES) if kind == "channel" else rng.choice(_PLANES[1:]), steps=rng.choice((1, 1, 5, 42)),
             dealias=0)
    if kind == "vortex":  # from 6 planes: w grows out of the z mode 2
        c["ny"] = c["nx"]
        c["dealias"] = rng.choice((0, 1)) if c["nz"] % 4 == 0 else 0  # 3 nz / 2 planes, an even number
    return c


# -- what a program has in hand before the call --------------------------------

_METHOD = {"direct": S.DIRECT, "mixed": S.MIXED, "pcg": S.JACPCG}


def _nodes(n, grading):
    """n elements on [0, 1], refined towards both ends by `grading`."""
    s = np.linspace(0.0, 1.0, n + 1)
    return s - grading * np.sin(2 * np.pi * s) / (2 * np.pi)


def _rect(d, c):
    tok = {"N_P": c["np"], "N_Z": c["nz"], "LAMBDA2": c["lambda2"], "BETA": 1.0, "TOL_REL": 1e-12}
    return sessions.rect_session(os.path.join(d, "case"), c["nx"], c["ny"], tokens=tok, fields="c",
                                 bcs={"w": {"c": "<D> 0.0"}}, xs=_nodes(c["nx"], c["grading"]),
                                 ys=_nodes(c["ny"], c["grading"]))


def _to_elements(a, nx, ny, np_):
    """Values on the mesh's distinct nodes [.., ny (np-1) + 1, nx (np-1) + 1]
    on its element nodes [.., ny nx, np, np]."""
    i = np.arange(nx)[:, None] * (np_ - 1) + np.arange(np_)
    j = np.arange(ny)[:, None] * (np_ - 1) + np.arange(np_)
    b = a[..., j[:, None, :, None], i[None, :, None, :]]
    return np.ascontiguousarray(b.reshape(a.shape[:-2] + (nx * ny, np_, np_)))


def _random_nodes(rng, c, planes):
    g = rng.uniform(-1.0, 1.0, (planes, c["ny"] * (c["np"] - 1) + 1, c["nx"] * (c["np"] - 1) + 1))
    return _to_elements(g, c["nx"], c["ny"], c["np"])


def _spectrum(rng, c):
    f = _random_nodes(rng, c, c["nz"])
    if c["nz"] > 1:
        f[1] = 0.0  # the Nyquist plane, which no solve touches
    return f


def _batch_problems(c):
    return sessions.uneven_batch(c["count"], c["problems"])


def _batch_case(p):
    return dict(nx=p["n"], ny=p["n"], np=p["np"], nz=1, grading=0.0, lambda2=p["lambda2"])


def _vortex_start(rng, x, y, z):
    a, b, g = rng.uniform(0, 2 * np.pi, 3)
    s = 1.0 + 0.1 * rng.uniform(-1, 1)
    z = np.asarray(z)[:, None, None, None]
    return {"u": s * np.sin(x + a)[None] * np.cos(y + b)[None] * np.cos(z + g),
            "v": -s * np.cos(x + a)[None] * np.sin(y + b)[None] * np.cos(z + g)}


def _dns_context(d, c):
    extra = {"DEALIAS": 1} if c["dealias"] else None
    path = os.path.join(d, "case")
    if c["flow"] == "vortex":
        sessions.taylor_green_session(path, c["nx"], c["np"], c["nz"], extra=extra)
    else:
        sessions.channel_session(path, c["nx"], c["ny"], c["np"], c["nz"], dt=2e-3, extra=extra)
    return S.Context(path)


def _dns_start(ctx, c, seed):
    x, y = ctx.mesh_coords()
    z = np.arange(ctx.nz) * 2 * np.pi / ctx.nz
    if c["flow"] == "vortex":
        ic = _vortex_start(np.random.default_rng(seed), x, y, z)
    else:
        ic = sessions.channel_initial(x, y, z, seed=seed, amplitude=0.05)
    zero = np.zeros((ctx.nz, ctx.nel, ctx.np, ctx.np))
    return {f: ic.get(f, zero) for f in ctx.fields}


def prepare(case, seed):
    c = case
    rng = np.random.default_rng(seed)
    st = {"kind": c["kind"]}
    with tempfile.TemporaryDirectory() as d:
        if c["kind"] in ("solve", "host", "grad"):
            ctx = S.Context(_rect(d, c))
            st["system"] = S.ModalMatrixSys(ctx, "c", c["lambda2"], method=_METHOD[c.get("method", "direct")])
            if c["kind"] == "solve":
                st["forcing"] = S.Field(ctx, "f").load_physical(_spectrum(rng, c))
                st["solution"] = S.Field(ctx, "c")
                st["pcg"] = c["method"] == "pcg"
            elif c["kind"] == "host":
                f = torch.from_numpy(_random_nodes(rng, c, c["nz"])).pin_memory()
                st["forcing"], st["solution"] = f.numpy(), torch.zeros_like(f).pin_memory().numpy()
            else:
                st["forcing"] = torch.from_numpy(_random_nodes(rng, c, c["nz"])).cuda().requires_grad_(True)
                st["seed"] = torch.from_numpy(rng.uniform(-1.0, 1.0, tuple(st["forcing"].shape))).cuda()
        elif c["kind"] == "batch":
            items = []
            for k, p in enumerate(_batch_problems(c)):
                pc = _batch_case(p)
                os.mkdir(os.path.join(d, str(k)))
                ctx = S.Context(_rect(os.path.join(d, str(k)), pc))
                items.append((S.ModalMatrixSys(ctx, "c", p["lambda2"]),
                              S.Field(ctx, "f").load_physical(_spectrum(rng, pc)), S.Field(ctx, "c")))
            st["batch"] = S.Batch(items)
        else:
            ctx = _dns_context(d, c)
            st["dns"] = S.DNS(ctx)
            ic = _dns_start(ctx, c, seed)
            if c["kind"] == "dns":
                # past the first-order start, well into the steady scheme
                st["dns"].restart(ic)
                st["dns"].advance(45)
                ctx.sync()
                st["steps"] = c["steps"]
            else:
                st["adjoint"] = S.DNSAdjoint(st["dns"], c["every"])
                st["steps"] = c["steps"]
                st["start"] = torch.from_numpy(np.stack([ic[f] for f in ctx.fields[:-1]])).cuda().requires_grad_(True)
                st["seed"] = torch.from_numpy(rng.uniform(-1.0, 1.0, tuple(st["start"].shape))).cuda()
    return st


# -- one pass ------------------------------------------------------------------


class _DeviceArray:
    """A library-owned device buffer for torch.as_tensor; `owner`, whose
    memory it is, lives as long as the tensor."""

    def __init__(self, ptr, shape, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": "<f8", "version": 3}


def _dns_fields(dns):
    """The fields of a DNS as they are held: device, Fourier space."""
    out = {}
    for f in dns.ctx.fields:
        p = ctypes.c_void_p()
        _lib.check(_lib.lib().stx_dns_field_ptr(dns._h, f.encode(), ctypes.byref(p)))
        out[f] = torch.as_tensor(_DeviceArray(p.value, (dns.ctx.nz, dns.ctx.plane_size), dns), device="cuda")
    return out


def run(state):
    st = state
    if st["kind"] == "solve":
        if st["pcg"]:
            st["solution"].data.zero_()  # the iteration starts from the field's values
            torch.cuda.current_stream().synchronize()
        return st["solution"].solve(st["forcing"], st["system"]).data
    if st["kind"] == "host":
        return st["system"].solve_host(st["forcing"], st["solution"])
    if st["kind"] == "grad":
        u = autograd.helmholtz_solve(st["forcing"], st["system"])
        return u.detach(), torch.autograd.grad(u, st["forcing"], st["seed"])[0]
    if st["kind"] == "batch":
        st["batch"].launch()
        return [u.data for _, _, u in st["batch"].items]
    if st["kind"] == "dns":
        st["dns"].advance(st["steps"])
        return _dns_fields(st["dns"])
    u = autograd.dns_steps(st["start"], st["adjoint"], st["steps"])
    return u.detach(), torch.autograd.grad(u, st["start"], st["seed"])[0]


# -- what a pass cannot do without -----------------------------------------------


def _solve_work(c):
    # forcing in, solution out; an element's fast diagonalisation (four small
    # matrix products) per plane
    n = c["nx"] * c["ny"] * c["np"] ** 2 * max(1, c["nz"] - 1)
    return 16.0 * n, 8.0 * c["np"] * n


def _dns_work(c):
    n = c["nx"] * c["ny"] * c["np"] ** 2 * c["nz"]
    ncom = 3 if c["nz"] > 1 else 2
    # three levels of velocity and nonlinear terms in (the newest nonlinear
    # term is formed), the new velocity, nonlinear term and pressure out
    nbytes = 8.0 * n * (5 * ncom + 2 * ncom + 1)
    # velocity gradients in two directions, the transforms, ncom + 1 solves
    flops = n * (ncom * 4 * c["np"] * 2 + 3 * ncom * 5 * math.log2(max(2, c["nz"])) + (ncom + 1) * 8 * c["np"])
    return nbytes, flops


def work(case):
    c = case
    if c["kind"] == "batch":
        b, f = (sum(v) for v in zip(*(_solve_work(_batch_case(p)) for p in _batch_problems(c))))
    elif c["kind"] in ("solve", "host"):
        b, f = _solve_work(c)
    elif c["kind"] == "grad":
        b, f = (2.0 * v for v in _solve_work(c))
    else:
        b, f = (v * c["steps"] for v in _dns_work(c))
        if c["kind"] == "adjoint":  # forward, recomputation and transposed steps
            b, f = 3.0 * b, 3.0 * f
    return {"bytes": b, "flops": f}


# -- the same results from plain numpy ---------------------------------------------
#
# On a rectangle of quads the assembled Helmholtz matrix is a sum of Kronecker
# products of one-dimensional matrices, so generalised eigenvectors of the two
# directions solve it for every constant.


def _gll(np_):
    """Gauss-Lobatto-Legendre points, weights and derivative matrix on [-1, 1]."""
    n = np_ - 1
    P = np.polynomial.legendre.Legendre.basis(n)
    z = np.concatenate([[-1.0], np.sort(P.deriv().roots().real), [1.0]])
    for _ in range(3):  # polish the interior roots of P'_n
        z[1:-1] -= P.deriv()(z[1:-1]) / P.deriv(2)(z[1:-1])
    p = P(z)
    w = 2.0 / (n * (n + 1) * p * p)
    D = np.zeros((np_, np_))
    for i in range(np_):
        for j in range(np_):
            if i != j:
                D[i, j] = p[i] / (p[j] * (z[i] - z[j]))
    D[0, 0], D[n, n] = -n * (n + 1) / 4.0, n * (n + 1) / 4.0
    return z, w, D


def _line(nodes, np_):
    """Eigenvalues and mass-orthonormal eigenvectors of the interior nodes of
    one direction, and the element masses [n, np]."""
    z, w, D = _gll(np_)
    n = len(nodes) - 1
    size = n * (np_ - 1) + 1
    K, m = np.zeros((size, size)), np.zeros(size)
    h = np.diff(nodes)
    for e in range(n):
        s = slice(e * (np_ - 1), e * (np_ - 1) + np_)
        K[s, s] += D.T @ (w[:, None] * D) * 2.0 / h[e]
        m[s] += w * h[e] / 2.0
    r = 1.0 / np.sqrt(m[1:-1])
    lam, V = np.linalg.eigh(r[:, None] * K[1:-1, 1:-1] * r[None, :])
    return lam, r[:, None] * V, w[None, :] * h[:, None] / 2.0


class _Rectangle:
    def __init__(self, c):
        self.c = c
        self.lx, self.Vx, mx = _line(_nodes(c["nx"], c["grading"]), c["np"])
        self.ly, self.Vy, my = _line(_nodes(c["ny"], c["grading"]), c["np"])
        self.mass = (my[:, None, :, None] * mx[None, :, None, :]).reshape(-1, c["np"], c["np"])

    def solve(self, f, const):
        """One plane of div grad u - const u = f on element nodes, u = 0 on the edges."""
        c = self.c
        q = c["np"] - 1
        g = np.zeros((c["ny"] * q + 1, c["nx"] * q + 1))
        b = (-self.mass * f).reshape(c["ny"], c["nx"], q + 1, q + 1)
        for j in range(c["ny"]):
            for i in range(c["nx"]):
                g[j * q : j * q + q + 1, i * q : i * q + q + 1] += b[j, i]
        h = self.Vy.T @ g[1:-1, 1:-1] @ self.Vx / (self.ly[:, None] + self.lx[None, :] + const)
        u = np.zeros_like(g)
        u[1:-1, 1:-1] = self.Vy @ h @ self.Vx.T
        return _to_elements(u, c["nx"], c["ny"], c["np"])

    def solve_spectrum(self, f):
        out = np.zeros_like(f)
        for k in range(self.c["nz"]):
            if self.c["nz"] == 1 or k != 1:
                out[k] = self.solve(f[k], self.c["lambda2"] + (k >> 1) ** 2)
        return out

    def solve_physical(self, f):
        nz = self.c["nz"]
        if nz == 1:
            return self.solve_spectrum(f)
        F = np.fft.rfft(f, axis=0) / nz
        U = np.zeros_like(F)
        for k in range((nz + 1) // 2):
            const = self.c["lambda2"] + k * k
            U[k] = self.solve(F[k].real, const) + 1j * self.solve(F[k].imag, const)
        return np.fft.irfft(U * nz, nz, axis=0)


def _planes(a, nz):
    """Element planes in the library's storage: rows of even length."""
    a = a.reshape(nz, -1)
    return torch.from_numpy(np.pad(a, ((0, 0), (0, a.shape[1] % 2))))


def exact(case, seed):
    c = case
    rng = np.random.default_rng(seed)
    if c["kind"] == "solve":
        return _planes(_Rectangle(c).solve_spectrum(_spectrum(rng, c)), c["nz"])
    if c["kind"] == "host":
        return _Rectangle(c).solve_physical(_random_nodes(rng, c, c["nz"]))
    if c["kind"] == "grad":
        R = _Rectangle(c)
        f = _random_nodes(rng, c, c["nz"])
        g = rng.uniform(-1.0, 1.0, f.shape)
        return R.solve_physical(f), R.mass * R.solve_physical(g / R.mass)
    if c["kind"] == "batch":
        cs = [_batch_case(p) for p in _batch_problems(c)]
        return [_planes(_Rectangle(p).solve_spectrum(_spectrum(rng, p)), 1) for p in cs]
    return None  # time stepping: the whole scheme would have to be written out again
