"""The output ring (z fastest) in the kernels that take it only from a size on: the persistent FP64 block
kernels beyond two wavelength tiles per SM, the mixed block and batch kernels beyond 56 MiB of outputs, and
the split solve's chain beyond 256 MiB.  The outputs equal the lambda-fastest ones (stored lane by lane) bit for bit
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
# by item with few and with many warps, staged
@pytest.mark.parametrize("nw,ncol", [(3, 3200), (33, 300), (5, 8000), (64, 150), (70, 101)])
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


def test_mixed_batch(engine):
    import numpy as np
    import torch

    from ocotillo_b200 import workloads
    rng = np.random.default_rng(6)
    kinds = [(n, int(w)) for n in list(range(2, 40)) + [64, 129] for w in rng.integers(1, 100, 2)]
    reps = (60 << 20) // (24 * sum(n * w for n, w in kinds)) + 1
    cols = {n: workloads.athena_column(n, rng, sigma_dex=0.3) for n in {n for n, _ in kinds}}
    nz, nw = (np.array([k[i] for k in kinds] * reps) for i in (0, 1))
    assert 24 * int((nz * nw).sum()) > 56 << 20
    grids = {w: workloads.log_wavelengths(w, 900.0, 40000.0) for w in set(nw.tolist())}
    at, pos = {}, 0
    for w, g in grids.items():
        at[w] = pos
        pos += len(g)
    rho, T = (torch.from_numpy(np.concatenate([cols[n][i] for n in nz.tolist()])).cuda() for i in (0, 1))
    dz = np.array([cols[n][2] for n in nz.tolist()])
    got = []
    for layout in (0, 1):
        b = engine.batch(nz, nw, dz, np.concatenate(list(grids.values())), np.array([at[w] for w in nw.tolist()]),
                         layout=layout, form="mixed")
        bufs = {}
        for k, v in b.alloc().items():
            buf = torch.full((v.numel() + 64,), -77.0, dtype=torch.float64, device="cuda")
            bufs[k] = (buf, buf[19:19 + v.numel()])
        b.bind(rho, T, {k: v[1] for k, v in bufs.items()})
        b.run()
        torch.cuda.synchronize()
        host = {}
        for k, (buf, view) in bufs.items():
            assert (buf[:19] == -77.0).all() and (buf[19 + view.numel():] == -77.0).all(), k
            host[k] = view.cpu()
        got.append([{k: b.column(host, i, k).contiguous().view(torch.int64) for k in KEYS} for i in range(len(nz))])
        b.close()
    for i, (x, y) in enumerate(zip(*got)):
        for k in KEYS:
            assert torch.equal(x[k], y[k]), (k, i, kinds[i % len(kinds)])
