"""Sums of the adjoint workload at the edges of their launch shapes: one
collect per layer over one to four tile sweeps, the streaming passes (diagonal
part of H, energy) at registers shorter than one round of their loads."""
import ctypes as C

import numpy as np
import pytest

from mettleq_b200.adjoint import AdjointEngine, LayeredAnsatz, PauliSum


def _product_state(n, rng, torch):
    """A normalised product state: its <P_q> are of order one at any size."""
    v = torch.ones(1, dtype=torch.complex128, device="cuda")
    for _ in range(n):
        z = rng.normal(size=2) + 1j * rng.normal(size=2)
        v = torch.kron(v, torch.tensor(z / np.linalg.norm(z), dtype=torch.complex128, device="cuda"))
    return v


@pytest.mark.gpu
@pytest.mark.parametrize("n,dtype", [(1, "complex64"), (2, "complex128"), (10, "complex64"), (11, "complex64"),
                                     (12, "complex64"), (12, "complex128"), (19, "complex64"), (19, "complex128"),
                                     (26, "complex64")])
def test_layer_values_and_energy(n, dtype):
    """Im <lam|X,Y,Z|psi> of every qubit, whatever the output held before,
    and E, H psi of a chain, against 64-bit torch."""
    import torch
    from mettleq_b200 import _native as N
    rng = np.random.default_rng(n)
    psi = _product_state(n, rng, torch)
    noise = torch.randn(1 << n, dtype=torch.complex128, device="cuda", generator=torch.Generator("cuda").manual_seed(n))
    lam = 1j * psi + 0.1 * noise / noise.norm()
    H = PauliSum.ising_chain(n, 0.8, -0.3)
    eng = AdjointEngine(LayeredAnsatz(n, 1), H, dtype=dtype)
    host = [x.cpu().numpy().astype(dtype) for x in (psi, lam)]
    psi, lam = (torch.tensor(x.astype(np.complex128), device="cuda") for x in host)
    # rounding of a thread's sum: its terms (at most 2^n / 2^15 amplitudes, 2^5 in small registers) * 2^-24
    tol = 1e-12 if dtype == "complex128" else 2.0 * max(32, 2 ** (n - 15)) * 2.0 ** -24
    try:
        eng.psi.set(host[0])
        eng.lam.set(host[1])
        qubits = np.arange(n, dtype=np.int32)
        mats = np.tile(np.array([1, 0, 0, 0, 0, 0, 1, 0], dtype=np.float64), n)
        got = torch.full((3 * n,), float("nan"), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        N.check(N.lib().mq_adjoint_layer_async(eng.psi.handle, eng.lam.handle, n, qubits.ctypes.data_as(C.c_void_p),
                                               mats.ctypes.data_as(C.c_void_p), C.c_void_p(got.data_ptr())))
        eng.psi.synchronize()
        got = got.cpu().numpy().reshape(n, 3)
        eng.psi.set(host[0])
        e = eng._pauli_sum()
        hpsi = torch.tensor(eng.lam.get().astype(np.complex128), device="cuda")
    finally:
        eng.close()
    want = np.empty((n, 3))
    ref = torch.zeros_like(psi)
    idx = torch.arange(1 << n, device="cuda")
    for q in range(n):
        p, l = psi.view(1 << q, 2, -1), lam.view(1 << q, 2, -1)
        x01 = torch.vdot(l[:, 0].reshape(-1), p[:, 1].reshape(-1)).item()
        x10 = torch.vdot(l[:, 1].reshape(-1), p[:, 0].reshape(-1)).item()
        z0 = torch.vdot(l[:, 0].reshape(-1), p[:, 0].reshape(-1)).item()
        z1 = torch.vdot(l[:, 1].reshape(-1), p[:, 1].reshape(-1)).item()
        want[q] = (x01 + x10).imag, (-1j * x01 + 1j * x10).imag, (z0 - z1).imag
        ref += -0.3 * p.flip(1).reshape(-1)
        if q + 1 < n:
            s = ((idx >> (n - 1 - q)) ^ (idx >> (n - 2 - q))) & 1
            ref += 0.8 * (1 - 2 * s).double() * psi
    assert np.max(np.abs(got - want)) < tol
    # lam is stored in the state's type: n + 1 roundings of terms that sum to at most 1.1 n |psi|
    eps = 2.0 ** -52 if dtype == "complex128" else 2.0 ** -23
    assert torch.max(torch.abs(hpsi - ref)).item() < (n + 2) * 1.1 * n * eps
    assert abs(e - torch.vdot(psi, hpsi).real.item()) < 1e-11 * n
