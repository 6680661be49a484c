"""The plane kernel (y inverse, x and y forward of one kz plane in shared memory)
against the oracle: the plain, filtered and Tungsten models (the Aluminum step is
in test_gpu_aluminum.py), both precisions, plane sides of every plan (powers of
two and mixed lengths, one line per turn up to several), the transform's own plane
and z kernels, and the reverse step.  Tolerances as in the other parity tests:
FP64 rounding over the steps, FP32 its own rounding level."""
import math

import numpy as np
import pytest

import openpfc_b200 as ob

pytestmark = pytest.mark.gpu

PI4 = [math.pi / 4] * 3
TOL = {ob.FP64: 1e-11, ob.FP32: 1e-5}
# (n0, n1, n2): smallest plane; mixed lengths on either side; turns of unequal
# length (65 columns); 512-point lines; a plane near the shared-memory limit
SHAPES = [(32, 16, 16), (48, 80, 16), (80, 24, 32), (192, 40, 16), (96, 96, 2), (128, 128, 16), (32, 512, 4),
          (512, 48, 8), (1024, 16, 4), (160, 48, 1), (64, 16, 40)]


@pytest.fixture(autouse=True)
def _plane(monkeypatch):
    monkeypatch.setenv("OPENPFC_GPU_AUTOTUNE_MODE", "fallback_only")
    monkeypatch.setenv("OPFC_PLANE", "1")


def _rel(a, b):
    return np.linalg.norm((a - b).ravel()) / np.linalg.norm(b.ravel())


@pytest.mark.parametrize("prec", [ob.FP64, ob.FP32])
@pytest.mark.parametrize("n", SHAPES)
def test_plain(oracle, n, prec):
    psi0 = ob.ic_noise(n, -0.285, 0.01, 3)
    m = ob.PfcB200(n, PI4, r=-0.25, precision=prec)
    m.initialize(0.5)
    m.set_psi(psi0)
    m.step(12)  # one graph of several steps, then single steps
    m.sync()
    assert _rel(m.get_psi(), oracle.run_plain(psi0, PI4, -0.25, 0.5, 12)) <= TOL[prec]
    # the captured steps read the mean of the field set last
    psi1 = ob.ic_noise(n, -0.2, 0.01, 4)
    m.set_psi(psi1)
    m.step(12)
    m.sync()
    assert _rel(m.get_psi(), oracle.run_plain(psi1, PI4, -0.25, 0.5, 12)) <= TOL[prec]


@pytest.mark.parametrize("prec", [ob.FP64, ob.FP32])
@pytest.mark.parametrize("n", [(32, 16, 16), (96, 40, 16), (64, 64, 16)])
def test_filtered_and_tungsten(oracle, n, prec):
    psi0 = ob.ic_noise(n, -0.10, 0.01, 5)
    m = ob.FilteredB200(n, PI4, r=-0.3, alpha=0.5, p2=-0.1, p3=-0.5, p4=0.3, precision=prec)
    m.initialize(0.5)
    m.set_psi(psi0)
    m.step(5)
    m.sync()
    ref = oracle.run_filtered(psi0, PI4, -0.3, 0.5, -0.1, -0.5, 0.3, 0.5, 5)
    assert _rel(m.get_psi(), ref) <= TOL[prec]
    dx = [1.1107207345395915] * 3
    psi0 = ob.ic_noise(n, -0.40, 0.01, 6)
    t = ob.TungstenB200(n, dx, precision=prec)
    t.initialize(1.0)
    t.set_psi(psi0)
    t.step(5)
    t.sync()
    assert _rel(t.get_psi(), oracle.run_tungsten(psi0, dx, oracle.TungstenParams.defaults(), 1.0, 5)) <= TOL[prec]


@pytest.mark.parametrize("n2", [1, 2, 16, 40, 48, 96, 256, 1024])
@pytest.mark.parametrize("prec", [ob.FP64, ob.FP32])
def test_transform_device_buffers(oracle, n2, prec):
    """Device buffers of the compute precision go straight through the kernels;
    an array off the complex boundary takes the copying path to the same values."""
    import torch

    n = (48, 16, n2)
    dt = torch.float64 if prec == ob.FP64 else torch.float32
    x = ob.ic_noise(n, 0.1, 1.0, 7)
    f = ob.B200Fft(n, precision=prec)
    ref = oracle.r2c(x)
    pad = torch.empty(x.size + 1, dtype=dt, device="cuda")
    for off in (0, 1):
        dev = pad[off:off + x.size].view(n2, 16, 48)
        dev.copy_(torch.from_numpy(x))
        hat = torch.empty((n2, 16, 25, 2), dtype=dt, device="cuda")
        torch.cuda.synchronize()
        f.forward(dev, hat)
        got = torch.view_as_complex(hat.double()).cpu().numpy()
        assert np.abs(got - ref).max() <= (1e-12 if prec == ob.FP64 else 2e-6) * np.abs(ref).max()
        back = torch.empty(x.size + 1, dtype=dt, device="cuda")[off:off + x.size].view(n2, 16, 48)
        f.backward(hat, back)
        torch.cuda.synchronize()
        assert np.abs(back.double().cpu().numpy() - x).max() <= (1e-12 if prec == ob.FP64 else 2e-6) * np.abs(x).max()


@pytest.mark.parametrize("prec,tol", [(ob.FP64, 1e-10), (ob.FP32, 1e-4)])
@pytest.mark.parametrize("n,z", [((32, 16, 32), None), ((48, 40, 48), None), ((64, 48, 80), None),
                                 ((32, 16, 256), 0), ((32, 16, 256), 6), ((32, 16, 256), 8), ((32, 16, 1024), 8),
                                 ((32, 16, 1024), 9)])
def test_adjoint_against_general_path(monkeypatch, n, z, prec, tol):
    """Two kernels a reverse step against the general reverse step (OPFC_PLANE=0):
    the same sums in another order, over 7 steps with segments of 3, 3 and 1.  The
    recomputation's z update reads one array and writes another, in the direct-load
    kernel (by default here) and in the pipelined ones (z forced)."""
    if z is not None:
        monkeypatch.setenv("OPFC_Z_VARIANT", str(z))
    psi0 = ob.ic_noise(n, -0.285, 0.05, 8)
    w = ob.ic_noise(n, 0.0, 1.0, 9)
    got = []
    for plane in ("1", "0"):
        monkeypatch.setenv("OPFC_PLANE", plane)
        m = ob.PfcB200(n, PI4, r=-0.25, precision=prec)
        m.initialize(0.5)
        m.set_psi(psi0)
        m.forward_checkpointed(7, 3)
        got.append(m.adjoint(w))
    (g1, r1, n1), (g0, r0, n0) = got
    assert _rel(np.asarray(g1), np.asarray(g0)) <= tol
    # dr and dn0 are sums with cancellation: relative to their terms' size
    assert abs(r1 - r0) <= tol * max(abs(r0), np.linalg.norm(w) * np.linalg.norm(psi0) * 1e-2)
    assert abs(n1 - n0) <= tol * max(abs(n0), np.abs(w).sum())


@pytest.mark.parametrize("plane", ["1", "0"])
def test_profile_and_nvtx_run_the_steps_kernels(monkeypatch, plane):
    """opfc_profile_step times what the step launches, and steps with NVTX ranges are
    the same steps (the plane kernel rounds differently from the passes)."""
    monkeypatch.setenv("OPFC_PLANE", plane)
    n = (64, 64, 48)
    psi0 = ob.ic_noise(n, -0.285, 0.01, 8)
    got = []
    for nvtx in ("0", "1"):
        monkeypatch.setenv("OPFC_NVTX", nvtx)
        m = ob.PfcB200(n, PI4, r=-0.25, precision=ob.FP32)
        m.initialize(0.5)
        m.set_psi(psi0)
        m.step(12)
        m.sync()
        got.append(m.get_psi())
    assert np.array_equal(*got)
    y = set() if plane == "1" else {"y_inverse", "y_forward"}
    assert set(m.profile_step(2)) == {"x_fused", "z_update", "hermitian_fix"} | y


@pytest.mark.parametrize("plane", ["1", "0"])
def test_adjoint_of_a_nonfinite_gradient(monkeypatch, plane):
    """Infinities in dLoss/dpsi_T come out as what they are: the non-finite flag
    reports the model's own field, which is finite here."""
    monkeypatch.setenv("OPFC_PLANE", plane)
    n = (32, 16, 32)
    m = ob.PfcB200(n, PI4, r=-0.25, precision=ob.FP64)
    m.initialize(0.5)
    m.set_psi(ob.ic_noise(n, -0.285, 0.01, 8))
    m.forward_checkpointed(3, 2)
    w = ob.ic_noise(n, 0.0, 1.0, 9)
    w[1, 2, 3] = np.inf
    g, _, _ = m.adjoint(w)
    assert not np.isfinite(g).all()
    m.step(1)
    m.sync()
    assert np.isfinite(m.get_psi()).all()


@pytest.mark.parametrize("prec", [ob.FP64, ob.FP32])
def test_ensemble(oracle, prec):
    sides = [(32, 16, 48), (48, 96, 16), (80, 48, 32), (128, 128, 16), (96, 80, 16), (64, 64, 64)]
    ms = [dict(n=s, dx=PI4, r=-0.2 - 0.02 * i) for i, s in enumerate(sides)]
    e = ob.Ensemble(ms, precision=prec)
    e.initialize(0.5)
    psi = [ob.ic_noise(s, -0.285 + 0.01 * i, 0.01, 10 + i) for i, s in enumerate(sides)]
    for i, p in enumerate(psi):
        e.set_psi(i, p)
    e.step(10)
    e.sync()
    for i, p in enumerate(psi):
        assert _rel(e.get_psi(i), oracle.run_plain(p, PI4, ms[i]["r"], 0.5, 10)) <= TOL[prec]


@pytest.fixture
def used_memory():
    """Small pieces of device memory that have held something before (bytes 0x40, as
    a double 32.5) and are free again, among others that are not."""
    import ctypes

    import torch

    torch.zeros(1, device="cuda")
    drv = ctypes.CDLL("libcuda.so.1")
    pieces = []
    for size in (512, 1024, 9480, 9480, 9480, 16384) * 64:
        p = ctypes.c_uint64()
        assert drv.cuMemAlloc_v2(ctypes.byref(p), ctypes.c_size_t(size)) == 0
        assert drv.cuMemsetD8_v2(p, ctypes.c_ubyte(0x40), ctypes.c_size_t(size)) == 0
        pieces.append(p)
    torch.cuda.synchronize()
    for p in pieces[::2]:
        assert drv.cuMemFree_v2(p) == 0
    yield
    for p in pieces[1::2]:
        assert drv.cuMemFree_v2(p) == 0


@pytest.mark.parametrize("plane", ["1", "0"])
@pytest.mark.parametrize("prec", [ob.FP64, ob.FP32])
def test_field_through_passes(oracle, monkeypatch, used_memory, plane, prec):
    """A field that came through opfc_pass keeps its mean in psi_hat, so the steps
    add none: also where the handle's memory held something before."""
    import torch

    from openpfc_b200.sharded import ARRAY_REAL, PASS_XY_FORWARD, PASS_Z_FORWARD, _CudaArray

    monkeypatch.setenv("OPFC_PLANE", plane)
    n = (32, 16, 48)
    psi0 = ob.ic_noise(n, -0.285, 0.01, 14)
    m = ob.PfcB200(n, PI4, r=-0.25, precision=prec)
    m.initialize(0.5)
    ptr = ob.lib().opfc_array(m.handle, ARRAY_REAL)
    real = torch.as_tensor(_CudaArray(ptr, m.shape, "<f8" if prec == ob.FP64 else "<f4"), device="cuda")
    real.copy_(torch.from_numpy(psi0))
    torch.cuda.synchronize()
    for p in (PASS_XY_FORWARD, PASS_Z_FORWARD):
        assert ob.lib().opfc_pass(m.handle, p, 0.0, 0) == 0
    m.step(3)
    m.sync()
    assert _rel(m.get_psi(), oracle.run_plain(psi0, PI4, -0.25, 0.5, 3)) <= TOL[prec]
