"""Differentiable permanents: output-pattern probabilities and log-likelihoods as
functions of the interferometer matrix or of its beam-splitter phases.

theboss has no derivatives.  d perm(U[T,S]) / d U[j][i] is T_j * S_i times the
(j, i) minor perm(U[T - e_j, S - e_i]); boss_perm_grad_batch returns all of them,
for every pattern, from one Glynn sweep per pattern (libboss_gb300.so).  Here
they back a torch.autograd.Function, and a Clements mesh (rectangular array of
m(m-1)/2 Mach-Zehnder interferometers, Clements et al., Optica 3, 1460 (2016))
maps phases to the unitary in torch so that gradients flow to the phases.
"""
from __future__ import annotations

import math
from functools import lru_cache
from typing import Sequence

import numpy as np
import torch

from . import _native


def _states(states, m: int) -> np.ndarray:
    a = np.asarray(states)
    if a.ndim == 1:
        a = a[None, :]
    if a.shape[1] != m:
        raise AttributeError("occupation vectors must have one entry per mode")
    return np.ascontiguousarray(np.rint(a).astype(np.int32))


class Permanents(torch.autograd.Function):
    """perms[k] = perm(U[T_k, S_k]); backward returns sum_k g_k * conj(d perm_k / dU),
    torch's convention for a holomorphic function of a complex tensor."""

    @staticmethod
    def forward(ctx, U: torch.Tensor, input_states: np.ndarray, output_states: np.ndarray):
        Un = np.ascontiguousarray(U.detach().cpu().numpy().astype(np.complex128))
        perms = _native.perm_batch(Un, input_states, output_states, _native.GLYNN)
        ctx.save_for_backward(U)
        ctx.states = (input_states, output_states)
        return torch.from_numpy(perms).to(U.device)

    @staticmethod
    def backward(ctx, grad_perms: torch.Tensor):
        (U,) = ctx.saved_tensors
        S, T = ctx.states
        Un = np.ascontiguousarray(U.detach().cpu().numpy().astype(np.complex128))
        _, grads = _native.perm_grad_batch(Un, S, T)
        g = torch.from_numpy(grads).to(U.device)
        gU = torch.einsum("k,kji->ji", grad_perms.to(g.dtype), g.conj())
        return gU, None, None


def permanents(U: torch.Tensor, input_states, output_states) -> torch.Tensor:
    m = U.shape[0]
    return Permanents.apply(U, _states(input_states, m), _states(output_states, m))


def _norms(input_states: np.ndarray, output_states: np.ndarray) -> np.ndarray:
    most = max(int(input_states.max(initial=0)), int(output_states.max(initial=0)))
    if most <= 20 and min(int(input_states.min(initial=0)), int(output_states.min(initial=0))) >= 0:
        table = np.array([math.factorial(k) for k in range(most + 1)], dtype=np.int64)  # 20! < 2^63
        f = table.__getitem__
    else:
        f = np.vectorize(math.factorial)
    return np.prod(f(input_states), axis=1).astype(np.float64) * np.prod(f(output_states), axis=1).astype(np.float64)


def probabilities(U: torch.Tensor, input_states, output_states) -> torch.Tensor:
    """|perm(U[T,S])|^2 / (prod S! prod T!) for every pattern."""
    m = U.shape[0]
    S, T = _states(input_states, m), _states(output_states, m)
    p = Permanents.apply(U, S, T)
    return (p.real ** 2 + p.imag ** 2) / torch.from_numpy(_norms(S, T)).to(p.real.device)


def log_likelihood(U: torch.Tensor, input_states, output_states) -> torch.Tensor:
    return torch.log(probabilities(U, input_states, output_states)).sum()


def clements_layers(m: int):
    """Mode pairs (k, k+1) of each layer of the rectangular mesh: even layers start
    at mode 0, odd layers at mode 1; m layers give m(m-1)/2 interferometers."""
    out = []
    for layer in range(m):
        start = layer % 2
        out.append(np.arange(start, m - 1, 2))
    return out


_DENSE_LAYERS = 96


@lru_cache(maxsize=8)
def _layer_entries(m: int):
    """Where each layer's non-zero entries lie in m stacked m x m matrices: the four
    entries of every interferometer (top-top, top-bottom, bottom-top, bottom-bottom,
    each over all layers), then the ones of the modes a layer leaves alone."""
    blocks, ones = [[], [], [], []], []
    for j, k in enumerate(clements_layers(m)):
        base = j * m * m
        for b, (r, c) in enumerate(((0, 0), (0, 1), (1, 0), (1, 1))):
            blocks[b].append(base + (k + r) * m + k + c)
        alone = np.setdiff1d(np.arange(m), np.concatenate([k, k + 1]))
        ones.append(base + alone * m + alone)
    ones = np.concatenate(ones)
    # arrays, not tensors: a tensor made while a call is traced would be the tracer's
    return np.concatenate([np.concatenate(b) for b in blocks] + [ones]), len(ones)


def _layer_product(theta: torch.Tensor, phi: torch.Tensor, m: int) -> torch.Tensor:
    """The mesh's layers applied one after the other."""
    ctype = torch.complex128
    M = torch.eye(m, dtype=ctype, device=theta.device)
    pos = 0
    for ks in clements_layers(m):
        k = torch.from_numpy(ks).to(theta.device)
        n = len(ks)
        th = theta[pos:pos + n]
        ep = torch.exp(1j * phi[pos:pos + n].to(ctype))
        pos += n
        c = torch.cos(th).to(ctype)
        s = torch.sin(th).to(ctype)
        top, bot = M[k], M[k + 1]
        new_top = (ep * c)[:, None] * top - s[:, None] * bot
        new_bot = (ep * s)[:, None] * top + c[:, None] * bot
        M = M.index_copy(0, k, new_top).index_copy(0, k + 1, new_bot)
    return M


def _dense_product(theta: torch.Tensor, phi: torch.Tensor, m: int) -> torch.Tensor:
    """The same from every layer as a dense m x m matrix, multiplied pairwise: 2 log2(m)
    batched products instead of some fifteen small operations per layer for autograd to
    follow."""
    ctype = torch.complex128
    ep, c, s = torch.exp(1j * phi.to(ctype)), torch.cos(theta).to(ctype), torch.sin(theta).to(ctype)
    at, ones = _layer_entries(m)
    v = torch.cat([ep * c, -s, ep * s, c, torch.ones(ones, dtype=ctype, device=theta.device)])
    L = torch.zeros(m * m * m, dtype=ctype, device=theta.device).index_copy(0, torch.from_numpy(at).to(theta.device), v)
    L = L.view(m, m, m)
    while L.shape[0] > 1:
        n = L.shape[0]
        P = L[1::2] @ L[0:n - n % 2:2]  # the later layer on the left
        L = torch.cat([P, L[-1:]]) if n % 2 else P
    return L[0]


def clements_unitary(theta: torch.Tensor, phi: torch.Tensor, output_phases: torch.Tensor = None) -> torch.Tensor:
    """U = D * T_L ... T_1 with T(theta, phi) on modes (k, k+1):
    [[e^{i phi} cos theta, -sin theta], [e^{i phi} sin theta, cos theta]]."""
    n_mzi = theta.shape[0]
    m = int(round((1 + math.sqrt(1 + 8 * n_mzi)) / 2))
    if m * (m - 1) // 2 != n_mzi or phi.shape[0] != n_mzi:
        raise ValueError("theta and phi need m(m-1)/2 entries each")
    ctype = torch.complex128
    if m <= _DENSE_LAYERS and torch.is_grad_enabled() and (theta.requires_grad or phi.requires_grad):
        # The derivatives of the dense layers' product, whose few operations autograd
        # follows in less time than the loop's (forward and backward, CPU: m = 24 8.3 -> 3.5 ms,
        # m = 96 72 -> 35; at m = 192 353 -> 282, with 113 MB in each of its m x m x m
        # steps: the line lies before that).  The value is the layers' own product, in
        # their order: derivatives of the logarithm of a small probability magnify the last
        # bits of U.
        dense = _dense_product(theta, phi, m)
        with torch.no_grad():
            value = _layer_product(theta.detach(), phi.detach(), m)
        M = value + (dense - dense.detach())
    else:
        M = _layer_product(theta, phi, m)
    if output_phases is not None:
        M = torch.exp(1j * output_phases.to(ctype))[:, None] * M
    return M
