"""Epilogue kernels at the edges of their tiles (1024 elements; 32 items x 32 levels; 16 levels; 32
columns x 32 wavelengths): random arrays, bit for bit against numpy's element operations, running
sum (cumsum) and in-order weighted sum."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", [0, 1])
@pytest.mark.parametrize("nx,ny,nz,nw", [(1, 1, 2, 1), (1, 1, 31, 40), (1, 3, 32, 11), (5, 7, 33, 1), (3, 11, 15, 33),
                                         (2, 16, 16, 32), (8, 5, 65, 13), (1, 129, 300, 3), (3, 1, 1030, 2)])
def test_sizes(layout, nx, ny, nz, nw):
    import torch
    from ocotillo_b200 import Engine, workloads
    rng = np.random.default_rng(nz * nw)
    ncol = nx * ny
    U, V = rng.standard_normal((nw, ncol, nz + 6)), rng.standard_normal((nw, ncol, nz))
    K = 10.0 ** rng.standard_normal((nw, ncol, nz))
    rho = 10.0 ** rng.standard_normal((ncol, nz))
    dz, target = 0.37, 0.2 * nz
    wa = workloads.log_wavelengths(nw)

    def dev(a):  # (nw, ncol, z) in the layout
        return torch.from_numpy(np.ascontiguousarray(a if layout == 0 else a.transpose(2, 1, 0))).cuda()

    def ref(t):
        a = t.cpu().numpy()
        return a.reshape(nw, ncol, nz) if layout == 0 else a.reshape(nz, ncol, nw).transpose(2, 1, 0)

    e = Engine(0)
    e.set_wavelengths(wa)
    u, v, k = dev(U), dev(V), dev(K)
    r = torch.from_numpy(rho).cuda()
    ip, im, tau = torch.empty_like(v), torch.empty_like(v), torch.empty_like(v)
    photo = torch.empty((nw, nx, ny), dtype=torch.int32, device="cuda")
    e.intensities_device(u, v, (nx, ny, nz), nw, {"Ip": ip, "Im": im}, layout=layout)
    e.optical_depth_device(k, r.view(nx, ny, nz), dz, target_tau=target, tau=tau, photo=photo, layout=layout)
    only = torch.empty_like(photo)
    e.optical_depth_device(k, r.view(nx, ny, nz), dz, target_tau=target, photo=only, layout=layout)
    plane = torch.from_numpy(np.ascontiguousarray(V[:, :, 0])).cuda()
    F = e.integrated_flux_device(plane, (nx, ny, nz))
    e.synchronize()
    torch.cuda.synchronize()
    assert np.array_equal(ref(ip), U[..., 3:-3] + V)
    assert np.array_equal(ref(im), U[..., 3:-3] - V)
    ref_tau = np.cumsum((K * rho[None]) * dz, axis=2)
    assert np.array_equal(ref(tau), ref_tau)
    reached = ref_tau >= target
    want = np.where(reached.any(axis=2), reached.argmax(axis=2), -1)
    assert np.array_equal(photo.cpu().numpy().reshape(nw, ncol), want)
    assert np.array_equal(only.cpu().numpy().reshape(nw, ncol), want)
    w = np.zeros(nw)
    for i in range(nw - 1):
        h = 0.5 * ((wa[i + 1] - wa[i]) * 1e-8)
        w[i] += h
        w[i + 1] += h
    f = np.zeros(ncol)
    for i in range(nw):
        f = f + w[i] * V[i, :, 0]
    assert np.array_equal(F.cpu().numpy().ravel(), f)
    # in place: tau over kappa, I+ over V
    e.optical_depth_device(k, r.view(nx, ny, nz), dz, tau=k, layout=layout)
    e.intensities_device(u, v, (nx, ny, nz), nw, {"Ip": v}, layout=layout)
    torch.cuda.synchronize()
    assert np.array_equal(ref(k), ref_tau) and np.array_equal(ref(v), U[..., 3:-3] + V)
    e.close()
