"""Differentiable Field::solve (the elliptic map forcing -> solution) and
DNS time steps (the discrete adjoint over the C ABI), as
torch.autograd.Functions.

Field::solve.  The map (src/field.cpp:598-809 with the z transforms of elliptic/helmholtz.cpp:
29-52) is affine, u = A f + b: b comes from the boundary conditions and
A = I S F, with F / I the packed real DFT pair and S, per plane, the
condensed Helmholtz solve S = -P H^-1 P^T M (P: global -> element-local
copy, H the symmetric assembled Helmholtz matrix of the plane's mode, M the
element-local mass Q4).  The packed DFT pair satisfies F^T = I W^-1 / N and
I^T = N W F with W = diag(1, 1, 2, 2, ...), a per-plane weight that commutes
with the per-plane S^T = -M P H^-1 P^T, and M commutes with the z transforms,
so
        A^T g = M (A (M^-1 g) - b)  =  Q4 * (solve(g / Q4) - solve(0)):
the gradient reuses the forward solve, its condensed factors included.
"""

from __future__ import annotations

import ctypes as C

import numpy as np

from . import FORWARD, INVERSE, JACPCG, _torch, solve_multi
from ._lib import check, lib


class _Work:
    """Device buffers and constants of one system, kept on the system: forcing
    and solution planes of one solve, and of the zero forcing beside it."""

    def __init__(self, system):
        torch = _torch()
        ctx = system.ctx
        self.F, self.U = ctx.new_field("adj_f"), ctx.new_field("adj_u")
        self.F0 = self.U0 = None
        self.reserved = system.method == JACPCG
        q4 = np.empty(ctx.nel * ctx.np * ctx.np)
        check(lib().stx_mesh_mass(ctx.handle, C.c_void_p(q4.ctypes.data)))
        self.q4 = torch.from_numpy(q4.reshape(1, ctx.nel, ctx.np, ctx.np)).to(self.F.data.device)
        torch.cuda.synchronize(self.F.data.device)

    def reserve(self, system):
        """Room for the backward pass's two fields from the forward one on: a
        first backward pass that grows the workspace takes 0.8 ms more."""
        if not self.reserved:
            check(lib().stx_modal_reserve(system.handle, 2))
            self.reserved = True

    def zero_pair(self, ctx):
        if self.F0 is None:
            self.F0, self.U0 = ctx.new_field("adj_f0"), ctx.new_field("adj_u0")
        return self.F0, self.U0


def _work(system):
    w = getattr(system, "_adjoint_work", None)
    if w is None:
        w = _Work(system)
        system._adjoint_work = w
    return w


def _solve(system, f, offset: bool):
    """solve(f), or with `offset` solve(f) - solve(0), as a new device tensor.

    The library's work and the copies around it run on the context stream,
    ordered after the caller's stream and before what that stream does next, by
    events: nothing is waited for on the host (eight device synchronisations a
    solve before: 12 x 12 x 32, N_P = 8, forward and backward 0.61 ms).  The
    result is allocated on the caller's stream; the work buffers belong to the
    system and are used on the context stream alone."""
    torch = _torch()
    ctx = system.ctx
    w = _work(system)
    n = ctx.nel * ctx.np * ctx.np
    shape = (ctx.nz, ctx.nel, ctx.np, ctx.np)
    if tuple(f.shape) != shape:
        raise ValueError(f"forcing shape {tuple(f.shape)} != {shape}")
    pairs = [(w.F, w.U)] + ([w.zero_pair(ctx)] if offset else [])
    device = w.F.data.device
    f = f.detach().reshape(ctx.nz, n)
    out = torch.empty(shape, dtype=torch.float64, device=device)
    caller, st = torch.cuda.current_stream(device), ctx.torch_stream()
    st.wait_stream(caller)
    try:
        with torch.cuda.stream(st):
            w.F.data[:, :n].copy_(f)
            w.F.transform(FORWARD)
            if ctx.nz > 1:  # the Nyquist planes, which a solve leaves alone
                w.F.data[1].zero_()
                for _, U in pairs:
                    U.data[1].zero_()
            if system.method == JACPCG:  # the iteration starts from zero
                for F, U in pairs:
                    U.data.zero_()
                    U.solve(F, system)
            elif offset:  # one pass over the matrices for both
                solve_multi([system] * 2, [F for F, _ in pairs], [U for _, U in pairs])
            else:
                w.U.solve(w.F, system)
            if offset:
                w.U.data.sub_(w.U0.data)
            w.U.transform(INVERSE)
            out.view(ctx.nz, n).copy_(w.U.data[:, :n])
    finally:  # f and out may be freed on the caller's stream, whatever happened
        caller.wait_stream(st)
    return out


def solve_physical(system, f):
    """u = Field::solve of the physical forcing f (device tensor [nz, nel, np, np],
    float64) with the system's BCs; returns a new device tensor."""
    return _solve(system, f, False)


def _helmholtz_solve():
    torch = _torch()

    class HelmholtzSolve(torch.autograd.Function):
        @staticmethod
        def forward(actx, f, system):
            actx.system = system
            if actx.needs_input_grad[0]:
                _work(system).reserve(system)
            return solve_physical(system, f)

        @staticmethod
        def backward(actx, g):
            system = actx.system
            w = _work(system)
            # less b = solve(0), the BC part of the affine map, taken afresh
            # each time: stx_field_bc_evaluate may have changed the BC values
            # (time-dependent BCs) since the forward call
            return w.q4 * _solve(system, g / w.q4, True), None

    return HelmholtzSolve


_FN = None


def helmholtz_solve(f, system):
    """Differentiable u = Field::solve(f) for a DIRECT (or MIXED) ModalMatrixSys."""
    global _FN
    if _FN is None:
        _FN = _helmholtz_solve()
    return _FN.apply(f, system)


def _dns_steps():
    torch = _torch()

    class DNSSteps(torch.autograd.Function):
        @staticmethod
        def forward(actx, u0, adjoint, nsteps, t0):
            dns = adjoint.dns
            a = u0.detach().to("cpu", torch.float64).numpy()
            dns.restart({c: a[i] for i, c in enumerate(adjoint.components)}, t0)
            adjoint.record(nsteps)
            out = np.stack([dns.field(c) for c in adjoint.components])
            actx.adjoint = adjoint
            actx.device = u0.device
            return torch.from_numpy(out).to(u0.device)

        @staticmethod
        def backward(actx, g):
            adj = actx.adjoint
            gn = g.detach().to("cpu", torch.float64).numpy()
            r = adj.backward({c: gn[i] for i, c in enumerate(adj.components)})
            grad = torch.from_numpy(np.stack([r[c] for c in adj.components])).to(actx.device)
            return grad, None, None, None

    return DNSSteps


_DNS_FN = None


def dns_steps(u0, adjoint, nsteps: int, t0: float = 0.0):
    """Differentiable final velocity of `nsteps` DNS time steps (integrate(),
    dns/integrate.cpp:138-200) from the initial velocity u0 (tensor
    [ncom, nz, nel, np, np], float64, physical; the DNS restarts from it at
    time t0 with empty history).  `adjoint` is a semtex_b200.DNSAdjoint of
    the DNS: the forward call records the run (checkpoints every
    checkpoint_every steps on the device), backward runs its discrete
    adjoint, whose solves reuse the step's condensed factors."""
    global _DNS_FN
    if _DNS_FN is None:
        _DNS_FN = _dns_steps()
    return _DNS_FN.apply(u0, adjoint, nsteps, t0)
