"""Columns whose levels share temperatures bit for bit (the floor of a disk) in every pattern the
FP64 sweep's kept factors distinguish, and operands outside the shared-reciprocal quotients' range:
block (both kernels), batch and no-allocation solves equal the oracle bit for bit.

Mixed form: the same columns against the stable FP64 form at the mixed form's tolerances, block and
batch bit for bit."""
import numpy as np
import pytest

from test_gpu_parity import assert_bitwise

pytestmark = pytest.mark.gpu

FIT = 2e4


@pytest.fixture(scope="module")
def engine():
    import torch
    assert torch.cuda.is_available()
    from ocotillo_b200 import Engine
    e = Engine(0)
    yield e
    e.close()


def _columns(nz, seed=3):
    """rho, T (8 columns of nz levels): one temperature; pairs; triples; alternating; a hot
    (ionized) plateau; a plateau that starts at the top, at the bottom; temperatures one ulp
    apart.  Densities vary per cell."""
    rng = np.random.default_rng(seed)
    z = np.arange(nz)
    T = np.empty((8, nz))
    T[0] = 2000.0
    T[1] = 3000.0 + 100.0 * (z // 2)
    T[2] = 8000.0 - 5.0 * (z // 3)
    T[3] = np.where(z % 2, 2000.0, 2500.0)
    T[4] = np.where(np.abs(z - nz // 2) < nz // 4, 3e4, 2000.0)
    T[5] = np.where(z > nz // 2, 2000.0, 5000.0 + z)
    T[6] = np.where(z < nz // 2, 2000.0, 5000.0 + z)
    T[7] = np.where(z % 3 == 0, np.nextafter(2000.0, 3000.0), 2000.0)
    rho = 1e-9 * np.exp(-0.5 * ((z - nz / 2) / (0.2 * nz)) ** 2)[None, :] * 10.0 ** (0.3 * rng.standard_normal((8, nz)))
    return rho.reshape(2, 4, nz), T.reshape(2, 4, nz)


@pytest.mark.parametrize("form", ["plain", "stable"])
@pytest.mark.parametrize("nz,nw", [(4, 40), (12, 33), (13, 64), (25, 96), (97, 5), (130, 70)])
def test_block_bitwise(engine, oracle, form, nz, nw):
    from ocotillo_b200 import workloads
    rho, T = _columns(nz)
    wa = workloads.log_wavelengths(nw)
    engine.set_wavelengths(wa)
    dz = 1e16 / (nz - 1)
    out = engine.solve_block(rho, T, dz, fully_ionized_T=FIT, form=form, allow_zero_pivot=True)
    ref = oracle.solve_block(rho, T, wa, dz, fully_ionized_T=FIT,
                             form=oracle.FORM_STABLE if form == "stable" else oracle.FORM_REFERENCE, backend="ocomath")
    for k in ("U", "kappa", "V"):
        assert_bitwise(out[k], ref[k], f"{form} {nz} {nw} {k}")


@pytest.mark.parametrize("form", ["plain", "stable"])
@pytest.mark.parametrize("scale,dz", [(1e-45, 1e13), (1e-70, 1e-3), (1e60, 1e13), (1e110, 1e-9), (1.0, 1e140), (1.0, 1e-150)])
def test_operands_out_of_range(engine, oracle, form, scale, dz):
    """Densities and spacings whose squares, ratios or products leave the range of the quotients
    from shared reciprocals (down to subnormal, up to overflowing)."""
    from ocotillo_b200 import workloads
    rho, T = _columns(20)
    rho = rho * scale
    wa = workloads.log_wavelengths(64)
    engine.set_wavelengths(wa)
    out = engine.solve_block(rho, T, dz, fully_ionized_T=FIT, form=form, allow_zero_pivot=True)
    ref = oracle.solve_block(rho, T, wa, dz, fully_ionized_T=FIT,
                             form=oracle.FORM_STABLE if form == "stable" else oracle.FORM_REFERENCE, backend="ocomath")
    assert out["zero_pivot"] == (ref["rc"] == -3)
    for k in ("U", "kappa", "V"):
        assert_bitwise(out[k], ref[k], f"{form} {scale} {dz} {k}")


@pytest.mark.parametrize("form", ["plain", "stable", "mixed"])
def test_batch_equals_block(engine, form):
    import torch

    from ocotillo_b200 import workloads
    rho, T = _columns(61)
    nz, nw = np.full(8, 61), np.array([40, 33, 64, 1, 96, 31, 32, 70])
    waves = [workloads.log_wavelengths(int(w)) for w in nw]
    off = np.concatenate([[0], np.cumsum(nw)[:-1]])
    dz = 1e16 / 60
    b = engine.batch(nz, nw, np.full(8, dz), np.concatenate(waves), off, fully_ionized_T=FIT, form=form)
    out = b.alloc()
    b.bind(torch.from_numpy(rho.ravel()).cuda(), torch.from_numpy(T.ravel()).cuda(), out)
    b.run()
    try:
        b.wait()
    except Exception as e:  # a zero pivot of the plain form is reported after every item is solved
        assert form == "plain" and "EZEROPIVOT" in str(e)
    for i in range(8):
        engine.set_wavelengths(waves[i])
        one = engine.solve_block(rho.reshape(8, 1, 1, 61)[i], T.reshape(8, 1, 1, 61)[i], dz, fully_ionized_T=FIT,
                                 form=form, allow_zero_pivot=True)
        for k in ("U", "kappa", "V"):
            assert_bitwise(b.column(out, i, k).cpu().numpy(), one[k][:, 0, 0, :].T, f"{form} column {i} {k}")
    b.close()


@pytest.mark.parametrize("nz,nw", [(21, 40), (130, 5)])
def test_mixed_against_stable(engine, nz, nw):
    from ocotillo_b200 import workloads
    rho, T = _columns(nz)
    engine.set_wavelengths(workloads.log_wavelengths(nw, 900.0, 40000.0))
    dz = 1e16 / (nz - 1)
    m = engine.solve_block(rho, T, dz, fully_ionized_T=FIT, form="mixed")
    s = engine.solve_block(rho, T, dz, fully_ionized_T=FIT, form="stable")
    for k, tol in (("kappa", 3e-5), ("U", 5e-4), ("Vtop", 1e-4), ("Vbot", 1e-4)):
        err = np.abs(m[k] / s[k] - 1.0).max()
        assert err <= tol, (k, err)
