"""The output ring (z fastest) in the block kernels that take it only from a size on: the persistent FP64
kernels beyond two wavelength tiles per SM, the mixed kernels beyond 56 MiB of outputs, and the split
solve's chain beyond 256 MiB.  The outputs equal the lambda-fastest ones (stored lane by lane) bit for bit
at every remainder of the groups of 8 levels, and nothing outside the arrays is written."""
import pytest

pytestmark = pytest.mark.gpu
KEYS = ("U", "kappa", "V")


@pytest.fixture(scope="module")
def engine():
    import torch
    assert torch.cuda.is_available()
    from ocotillo_b200 import Engine
    e = Engine(0)
    yield e
    e.close()


def _check(engine, ncol, nz, nw, form, grey=False):
    """ncol columns that repeat 16 different ones."""
    import torch

    from ocotillo_b200 import workloads
    if not grey:
        engine.set_wavelengths(workloads.log_wavelengths(nw, 900.0, 40000.0))
    rho, T, dz = workloads.agn_block(1, 16, nz, seed=nz)
    idx = torch.arange(ncol, device="cuda") % 16
    r, t = (torch.from_numpy(x).cuda()[:, idx].contiguous() for x in (rho, T))
    rows = {"U": nz + 6, "kappa": nz, "V": nz}
    shift = nz % 8
    ref, lam = {}, {}
    for k, n in rows.items():
        buf = torch.full((nw * ncol * n + 64,), -77.0, dtype=torch.float64, device="cuda")
        ref[k] = (buf, buf[16 + shift:16 + shift + nw * ncol * n])
        lam[k] = torch.empty((n, ncol, nw), dtype=torch.float64, device="cuda")
    engine.solve_block_device(r, t, dz, {k: v[1] for k, v in ref.items()}, form=form, layout=0, lgrey=grey)
    engine.solve_block_device(r, t, dz, lam, form=form, layout=1, lgrey=grey)
    torch.cuda.synchronize()
    for k, n in rows.items():
        buf, view = ref[k]
        assert (buf[:16 + shift] == -77.0).all() and (buf[16 + shift + view.numel():] == -77.0).all(), (k, nz)
        a = view.view(nw, ncol, n).view(torch.int64)
        assert torch.equal(a, lam[k].permute(2, 1, 0).contiguous().view(torch.int64)), (k, nz)


def _pivots(engine, form):
    try:
        engine.synchronize()
    except Exception as e:  # a zero pivot of the plain form
        assert form == "plain" and "EZEROPIVOT" in str(e)


@pytest.mark.parametrize("form", ["plain", "stable"])
@pytest.mark.parametrize("nw,ncol", [(3, 3200), (33, 300), (64, 150), (70, 101)])  # by item, by item, staged, staged
def test_persistent(engine, form, nw, ncol):
    for nz in list(range(2, 36)) + [63, 64, 65, 100]:
        _check(engine, ncol, nz, nw, form)
    _pivots(engine, form)


@pytest.mark.parametrize("nw", [3, 33, 64, 70])
def test_mixed(engine, nw):
    for nz in list(range(2, 21)) + [31, 32, 33, 64, 100]:
        _check(engine, (57 << 20) // (24 * nz * nw) + 33, nz, nw, "mixed")
    _pivots(engine, "mixed")


@pytest.mark.parametrize("form", ["plain", "stable"])
@pytest.mark.parametrize("ncol,nw,nz0,grey", [(148, 64, 1190, False), (1890, 5, 1192, False), (16395, 1, 690, True)])
def test_split_chain(engine, form, ncol, nw, nz0, grey):
    for nz in range(nz0, nz0 + 8):
        _check(engine, ncol, nz, nw, form, grey)
    _pivots(engine, form)
