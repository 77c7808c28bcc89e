"""The persistent FP64 kernels (blocks beyond two wavelength tiles per SM, ragged batches, the solve without
allocations) on the columns and operands that test_gpu_plateau gives the split solve: levels that share
temperatures in every pattern, and densities and spacings whose squares, ratios or products leave the range
of the quotients from shared reciprocals.  Equal to the oracle bit for bit, in both layouts."""
import ctypes

import numpy as np
import pytest

from test_gpu_parity import assert_bitwise
from test_gpu_plateau import FIT, _columns

pytestmark = pytest.mark.gpu
OPERANDS = [(1e-45, 1e13), (1e-70, 1e-3), (1e60, 1e13), (1e110, 1e-9), (1.0, 1e140), (1.0, 1e-150)]


@pytest.fixture(scope="module")
def engine():
    import torch
    assert torch.cuda.is_available()
    from ocotillo_b200 import Engine
    e = Engine(0)
    yield e
    e.close()


def _reference(oracle, rho, T, wa, dz, form):
    return oracle.solve_block(rho.reshape(8, 1, -1), T.reshape(8, 1, -1), wa, dz, fully_ionized_T=FIT,
                              form=oracle.FORM_STABLE if form == "stable" else oracle.FORM_REFERENCE, backend="ocomath")


def _check(engine, oracle, rho, T, dz, nw, form, items=0):
    import torch

    from ocotillo_b200 import workloads
    nz = rho.shape[-1]
    wa = workloads.log_wavelengths(nw)
    ref = _reference(oracle, rho, T, wa, dz, form)
    tiles = (nw + 31) // 32 if nw >= 64 or nw % 32 == 0 else nw / 32
    rep = max(int(297 / tiles / 8), items // (8 * nw)) + 1  # copies of the 8 columns
    r, t = (torch.from_numpy(x.reshape(1, 8, nz)).cuda().repeat(1, rep, 1) for x in (rho, T))
    engine.set_wavelengths(wa)
    for layout in (0, 1):
        out = {k: torch.empty(nw * 8 * rep * (nz + 6 * (k == "U")), dtype=torch.float64, device="cuda") for k in ("U", "kappa", "V")}
        n0 = engine.kernel_launches
        engine.solve_block_device(r, t, dz, out, fully_ionized_T=FIT, form=form, layout=layout)
        assert engine.kernel_launches - n0 == 2  # records and one solve kernel
        try:
            engine.synchronize()
            zero = False
        except Exception as e:
            assert "EZEROPIVOT" in str(e)
            zero = True
        assert zero == (ref["rc"] == -3)
        for k, v in out.items():
            n = nz + 6 * (k == "U")
            a = v.view(nw, rep, 8, n) if layout == 0 else v.view(n, rep, 8, nw).permute(3, 1, 2, 0)
            a = a.contiguous().cpu().numpy()
            for i in range(rep):
                assert_bitwise(a[:, i], ref[k][:, :, 0, :], f"{form} {nw} layout {layout} copy {i} {k}")


@pytest.mark.parametrize("form", ["plain", "stable"])
@pytest.mark.parametrize("nz,nw", [(4, 40), (13, 64), (25, 96), (97, 5), (130, 70)])
def test_plateaus(engine, oracle, form, nz, nw):
    rho, T = _columns(nz)
    _check(engine, oracle, rho, T, 1e16 / (nz - 1), nw, form)


@pytest.mark.parametrize("form", ["plain", "stable"])
@pytest.mark.parametrize("nw", [33, 64])
@pytest.mark.parametrize("scale,dz", OPERANDS)
def test_operands_out_of_range(engine, oracle, form, nw, scale, dz):
    rho, T = _columns(20)
    _check(engine, oracle, rho * scale, T, dz, nw, form)


@pytest.mark.parametrize("form", ["plain", "stable"])
@pytest.mark.parametrize("nz,nw", [(4, 40), (13, 33), (60, 40)])
def test_more_warps_than_two_blocks_per_sm_hold(engine, oracle, form, nz, nw):
    """The by-item kernel's variant for many warps (three blocks per SM)."""
    rho, T = _columns(nz)
    _check(engine, oracle, rho, T, 1e16 / (nz - 1), nw, form, items=148 * 2 * 128)


@pytest.mark.parametrize("form", ["plain", "stable"])
@pytest.mark.parametrize("scale,dz", OPERANDS)
def test_batch_and_noalloc(engine, oracle, form, scale, dz):
    import torch

    from ocotillo_b200 import workloads
    from ocotillo_b200.engine import _DP, load_library
    rho, T = _columns(20)
    rho = rho * scale
    lib = load_library()
    dr, dt = torch.from_numpy(rho).cuda(), torch.from_numpy(T).cuda()
    for nw in (33, 64):
        wa = np.ascontiguousarray(workloads.log_wavelengths(nw))
        ref = _reference(oracle, rho, T, wa, dz, form)
        for layout in (0, 1):
            b = engine.batch(np.full(8, 20), np.full(8, nw), np.full(8, dz), wa, np.zeros(8, dtype=np.int64),
                             fully_ionized_T=FIT, form=form, layout=layout)
            out = b.alloc()
            b.bind(dr.view(-1), dt.view(-1), out)
            b.run()
            torch.cuda.synchronize()
            for k in ("U", "kappa", "V"):
                for i in range(8):
                    a = b.column(out, i, k).cpu().numpy()
                    assert_bitwise(a.T, ref[k][:, i, 0, :], f"batch {form} {nw} {layout} {i} {k}")
            b.close()
            n = {"U": 26, "kappa": 20, "V": 20}
            got = {k: torch.empty(nw * 8 * m, dtype=torch.float64, device="cuda") for k, m in n.items()}
            prm = engine.params((2, 4, 20), nw, dz, fully_ionized_T=FIT, form=form, layout=layout)
            ptr = lambda x: ctypes.c_void_p(x.data_ptr())
            rc = lib.oco_solve_block_noalloc(ctypes.byref(prm), wa.ctypes.data_as(_DP), ptr(dr), ptr(dt), ptr(got["U"]),
                                             ptr(got["kappa"]), ptr(got["V"]), None, None,
                                             ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
            assert rc == ref["rc"]
            for k, m in n.items():
                a = got[k].view(nw, 8, m) if layout == 0 else got[k].view(m, 8, nw).permute(2, 1, 0)
                assert_bitwise(a.contiguous().cpu().numpy(), ref[k][:, :, 0, :], f"noalloc {form} {nw} {layout} {k}")
