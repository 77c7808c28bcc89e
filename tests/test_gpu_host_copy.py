"""Host-array block solves into pageable and pinned arrays, in one chunk and in several, with
outputs below and above the pinned slots' sizes, and from two threads at once, equal the device-array
solve bit for bit."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
KEYS = ("U", "kappa", "V", "Vtop", "Vbot")


def _device(shape, nw, seed):
    import torch
    from ocotillo_b200 import Engine, workloads
    rho, T, dz = workloads.agn_block(*shape, seed=seed)
    wa = workloads.log_wavelengths(nw)
    e = Engine(0)
    e.set_wavelengths(wa)
    nx, ny, nz = shape
    dims = {"U": (nw, nx, ny, nz + 6), "kappa": (nw, nx, ny, nz), "V": (nw, nx, ny, nz), "Vtop": (nw, nx, ny),
            "Vbot": (nw, nx, ny)}
    out = {k: torch.empty(d, dtype=torch.float64, device="cuda") for k, d in dims.items()}
    e.solve_block_device(torch.from_numpy(rho).cuda(), torch.from_numpy(T).cuda(), dz, out, form="stable")
    e.synchronize()
    ref = {k: v.cpu().numpy() for k, v in out.items()}
    e.close()
    return rho, T, dz, wa, dims, ref


def _equal(a, ref):
    for k in a:
        if k in ref:
            assert np.array_equal(a[k].view(np.uint64), ref[k].view(np.uint64)), k


@pytest.mark.parametrize("gb", [None, "0.004"])
@pytest.mark.parametrize("shape,nw", [((5, 7, 33), 3), ((9, 11, 65), 17), ((16, 20, 100), 40)])
def test_pageable_and_pinned(monkeypatch, gb, shape, nw):
    import torch
    from ocotillo_b200 import Engine
    rho, T, dz, wa, dims, ref = _device(shape, nw, 3)
    if gb:
        monkeypatch.setenv("OCO_WORKSPACE_GB", gb)
    e = Engine(0)
    e.set_wavelengths(wa)
    _equal(e.solve_block(rho, T, dz, form="stable"), ref)
    pinned = {k: torch.empty(dims[k], dtype=torch.float64, pin_memory=True).numpy() for k in ("U", "Vtop")}
    _equal(e.solve_block(rho, T, dz, form="stable", out=pinned), ref)
    _equal(e.solve_block(rho, T, dz, form="stable", want=("V",)), ref)
    # a view of a larger array: nothing outside it is written
    big = np.full(ref["kappa"].size + 64, -7.0)
    view = big[32:-32].reshape(dims["kappa"])
    _equal(e.solve_block(rho, T, dz, form="stable", want=("kappa",), out={"kappa": view}), ref)
    assert (big[:32] == -7.0).all() and (big[-32:] == -7.0).all()
    e.close()


def test_two_threads():
    from ocotillo_b200 import Engine
    cases = [_device((12, 13, 70), 24, s) for s in (4, 5)]
    bad = []

    def work(case):
        try:
            rho, T, dz, wa, dims, ref = case
            e = Engine(0)
            e.set_wavelengths(wa)
            for _ in range(5):
                _equal(e.solve_block(rho, T, dz, form="stable"), ref)
            e.close()
        except BaseException as x:  # reported by the main thread
            bad.append(x)

    th = [threading.Thread(target=work, args=(c,)) for c in cases]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not bad, bad
