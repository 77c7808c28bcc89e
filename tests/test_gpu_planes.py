"""Solves that ask for the emergent planes alone (nothing stored per level, kappa of the two ends
only, back-substitution without fluxes down to the bottom's last levels) give the planes of the full
solve bit for bit, at every remainder of the sweeps' groups."""
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


@pytest.mark.parametrize("form", ["plain", "stable", "mixed"])
@pytest.mark.parametrize("ncol,nw", [(3, 5), (2, 70), (5, 2048)])  # by item, few tiles, many tiles
def test_block(engine, form, ncol, nw):
    import torch

    from ocotillo_b200 import workloads
    engine.set_wavelengths(workloads.log_wavelengths(nw))
    for nz in list(range(2, 24)) + [47, 48, 49, 64, 90, 91, 97]:
        rho, T, dz = workloads.agn_block(1, ncol, nz, seed=nz, rho_floor=1e-15)
        r, t = torch.from_numpy(rho).cuda(), torch.from_numpy(T).cuda()
        mk = lambda *s: torch.full(s, -3.0, dtype=torch.float64, device="cuda")
        full = {"U": mk(nz + 6, ncol, nw), "kappa": mk(nz, ncol, nw), "V": mk(nz, ncol, nw), "Vtop": mk(nw, 1, ncol),
                "Vbot": mk(nw, 1, ncol)}
        planes = {"Vtop": mk(nw, 1, ncol), "Vbot": mk(nw, 1, ncol)}
        engine.solve_block_device(r, t, dz, full, form=form, layout=1)
        engine.solve_block_device(r, t, dz, planes, form=form, layout=nz % 2)
        torch.cuda.synchronize()
        for k in planes:
            a, b = planes[k].cpu().numpy(), full[k].cpu().numpy()
            assert np.array_equal(a.view(np.uint64), b.view(np.uint64)), (k, nz)
        v = full["V"].cpu().numpy()
        assert np.array_equal(v[-1].T.ravel().view(np.uint64), planes["Vtop"].cpu().numpy().ravel().view(np.uint64))
        assert np.array_equal(v[0].T.ravel().view(np.uint64), planes["Vbot"].cpu().numpy().ravel().view(np.uint64))
    try:
        engine.synchronize()
    except Exception as e:  # a zero pivot of the plain form
        assert form == "plain" and "EZEROPIVOT" in str(e)


@pytest.mark.parametrize("form", ["plain", "stable", "mixed"])
def test_batch(engine, form):
    import torch

    from ocotillo_b200 import workloads
    rng = np.random.default_rng(8)
    nz = np.array(list(range(2, 30)) + [50, 51, 130])
    nw = rng.integers(1, 90, len(nz))
    waves = [workloads.log_wavelengths(int(w), 900.0, 40000.0) for w in nw]
    off = np.concatenate([[0], np.cumsum(nw)[:-1]])
    cols = [workloads.athena_column(int(n), rng, sigma_dex=0.3) for n in nz]
    rho = torch.from_numpy(np.concatenate([c[0] for c in cols])).cuda()
    T = torch.from_numpy(np.concatenate([c[1] for c in cols])).cuda()
    got = []
    for want in (("U", "kappa", "V", "Vtop", "Vbot"), ("Vtop", "Vbot")):
        b = engine.batch(nz, nw, np.array([c[2] for c in cols]), np.concatenate(waves), off, form=form)
        out = b.alloc(want=want)
        b.bind(rho, T, out)
        b.run()
        torch.cuda.synchronize()
        got.append({k: out[k].cpu().numpy() for k in ("Vtop", "Vbot")})
        b.close()
    for k in got[0]:
        assert np.array_equal(got[0][k].view(np.uint64), got[1][k].view(np.uint64)), k
