"""The reference layout's outputs (z fastest, written in 64-byte runs through a ring of levels)
equal the lambda-fastest ones (stored lane by lane) bit for bit, at every alignment of the rows and
every remainder of the groups of 8 levels, and nothing outside the arrays is written."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine():
    import torch
    assert torch.cuda.is_available()
    from ocotillo_b200 import Engine
    e = Engine(0)
    yield e
    e.close()


def _guarded(n, shift):
    """n elements inside a filled buffer, shift elements past its (256-byte aligned) start."""
    import torch
    buf = torch.full((n + 64,), -77.0, dtype=torch.float64, device="cuda")
    return buf, buf[16 + shift:16 + shift + n]


def _check_guards(bufs, shift):
    for buf, view in bufs.values():
        g = buf.cpu().numpy()
        n = view.numel()
        assert (g[:16 + shift] == -77.0).all() and (g[16 + shift + n:] == -77.0).all()


@pytest.mark.parametrize("form", ["plain", "stable", "mixed"])
@pytest.mark.parametrize("nw", [3, 33, 64])
def test_block(engine, form, nw):
    import torch

    from ocotillo_b200 import workloads
    engine.set_wavelengths(workloads.log_wavelengths(nw, 900.0, 40000.0))
    for nz in list(range(2, 36)) + [63, 64, 65, 100]:
        rho, T, dz = workloads.agn_block(1, 5, nz, seed=nz)
        r, t = torch.from_numpy(rho).cuda(), torch.from_numpy(T).cuda()
        n = {"U": nw * 5 * (nz + 6), "kappa": nw * 5 * nz, "V": nw * 5 * nz, "Vtop": nw * 5, "Vbot": nw * 5}
        shift = nz % 8
        ref = {k: _guarded(v, shift) for k, v in n.items()}
        lam = {k: torch.empty(v, dtype=torch.float64, device="cuda") for k, v in n.items()}
        engine.solve_block_device(r, t, dz, {k: v[1] for k, v in ref.items()}, form=form, layout=0)
        engine.solve_block_device(r, t, dz, lam, form=form, layout=1)
        torch.cuda.synchronize()
        _check_guards(ref, shift)
        for k in ("U", "kappa", "V"):
            rows = nz + 6 if k == "U" else nz
            a = ref[k][1].view(nw, 5, rows).cpu().numpy()
            b = lam[k].view(rows, 5, nw).cpu().numpy().transpose(2, 1, 0)
            assert np.array_equal(a.view(np.uint64), np.ascontiguousarray(b).view(np.uint64)), (k, nz)
        for k in ("Vtop", "Vbot"):
            assert np.array_equal(ref[k][1].cpu().numpy().view(np.uint64), lam[k].cpu().numpy().view(np.uint64)), (k, nz)
    try:
        engine.synchronize()
    except Exception as e:  # a zero pivot of the plain form
        assert form == "plain" and "EZEROPIVOT" in str(e)


@pytest.mark.parametrize("form", ["plain", "stable", "mixed"])
def test_batch(engine, form):
    import torch

    from ocotillo_b200 import workloads
    rng = np.random.default_rng(5)
    nz = np.array(list(range(2, 40)) + [64, 129])
    nw = rng.integers(1, 70, len(nz))
    waves = [workloads.log_wavelengths(int(w), 900.0, 40000.0) for w in nw]
    off = np.concatenate([[0], np.cumsum(nw)[:-1]])
    cols = [workloads.athena_column(int(n), rng, sigma_dex=0.3) for n in nz]
    rho = torch.from_numpy(np.concatenate([c[0] for c in cols])).cuda()
    T = torch.from_numpy(np.concatenate([c[1] for c in cols])).cuda()
    dz = np.array([c[2] for c in cols])
    out = []
    for layout in (0, 1):
        b = engine.batch(nz, nw, dz, np.concatenate(waves), off, layout=layout, form=form)
        bufs = {k: _guarded(v.numel(), 3) for k, v in b.alloc().items()}
        b.bind(rho, T, {k: v[1] for k, v in bufs.items()})
        b.run()
        torch.cuda.synchronize()
        _check_guards(bufs, 3)
        out.append([{k: b.column({n: v[1] for n, v in bufs.items()}, i, k).cpu().numpy() for k in bufs} for i in range(len(nz))])
        b.close()
    for i, (x, y) in enumerate(zip(*out)):
        for k in x:
            assert np.array_equal(np.ascontiguousarray(x[k]).view(np.uint64), np.ascontiguousarray(y[k]).view(np.uint64)), (k, i)
