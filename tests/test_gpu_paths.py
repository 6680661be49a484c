"""Every kernel that a step may take against the oracle: the defaults, and each
variant of the separate passes (persistent TMA/bulk-copy-fed and direct loads)
forced, for the plain, filtered and Tungsten models in both precisions."""
import math

import numpy as np
import pytest

import openpfc_b200 as ob

pytestmark = pytest.mark.gpu

PI4 = [math.pi / 4] * 3


# the y, x and z variants of each path (OPFC_Y_VARIANT, ...), all as separate passes
PATHS = {"tma": (0, 0, 0), "tma_radial": (0, 0, 1), "direct": (0, 0, 0), "direct_xyz": (1, 1, 2),
         "computed": (2, 2, 3), "direct_computed": (0, 0, 4), "pingpong": (3, 3, 5), "e32": (4, 0, 0),
         "folded": (3, 3, 6), "folded_direct": (0, 0, 7), "folded_nopp": (0, 4, 8), "folded_wide": (0, 0, 9)}


@pytest.fixture(params=["default"] + list(PATHS))
def path(request, monkeypatch):
    """default: what a handle takes by itself (the plane kernel on small grids);
    tma: pipelined kernels streaming the per-mode tables;
    tma_radial: the z update reading radial operator tables (isotropic grids;
    others fall back to tables);
    direct: direct-load kernels (OPFC_NO_TMA=1);
    direct_xyz: the direct-load variants of the three passes;
    computed: pipelined z update computing its operators from k^2, half-width y
    tiles and the x pass without the warp-square kernel;
    direct_computed: direct z update computing its operators;
    pingpong: ping-pong FFT exchange buffers in the y pass and the computed z
    update, and the x pass's warp-square kernel with rows loaded straight into
    registers;
    e32: direct-load y pass with 32 values per thread (other lengths keep their plan);
    folded: the z update reading the folded FP64-built tables with ping-pong
    exchange buffers, with the ping-pong y pass and the register-loaded x pass;
    folded_direct: direct-load z update on the folded tables;
    folded_nopp: pipelined z update on the folded tables without ping-pong buffers
    with the register-loaded x pass prefetching the next row;
    folded_wide: the z update on the folded tables with 128-byte tile rows
    streamed through a two-slot box ring (z lengths other than 1024 and the
    Tungsten model take the direct-load kernel).
    The Tungsten model has no computed operators and falls back to tables."""
    for k in ("OPFC_NO_TMA", "OPFC_PLANE", "OPFC_Y_VARIANT", "OPFC_X_VARIANT", "OPFC_Z_VARIANT"):
        monkeypatch.delenv(k, raising=False)
    monkeypatch.setenv("OPENPFC_GPU_AUTOTUNE_MODE", "fallback_only")
    if request.param == "direct":
        monkeypatch.setenv("OPFC_NO_TMA", "1")
    if request.param != "default":
        monkeypatch.setenv("OPFC_PLANE", "0")
        for k, v in zip(("OPFC_Y_VARIANT", "OPFC_X_VARIANT", "OPFC_Z_VARIANT"), PATHS[request.param]):
            monkeypatch.setenv(k, str(v))
    return request.param


def rel_l2(a, b):
    return float(np.linalg.norm((a - b).ravel()) / np.linalg.norm(b.ravel()))


@pytest.mark.parametrize("prec,tol", [(ob.FP64, 1e-11), (ob.FP32, 1e-5)])
@pytest.mark.parametrize("n", [(64, 64, 64), (128, 32, 256), (256, 16, 512), (512, 32, 16), (1024, 16, 16),
                               (16, 512, 512), (32, 128, 128), (32, 16, 1024), (32, 1024, 16)])
def test_plain(oracle, path, prec, tol, n):
    psi0 = oracle.ic_noise(n, -0.285, 0.01, 3)
    ref = oracle.run_plain(psi0, PI4, -0.25, 0.5, 10)
    m = ob.PfcB200(n, PI4, precision=prec)
    m.initialize(0.5)
    m.set_psi(psi0)
    m.step(10)
    m.sync()
    assert rel_l2(m.get_psi(), ref) <= tol


@pytest.mark.parametrize("prec,tol", [(ob.FP64, 1e-11), (ob.FP32, 1e-5)])
@pytest.mark.parametrize("n", [(64, 64, 32), (512, 16, 16), (128, 32, 32), (1024, 16, 8), (16, 32, 1024)])
def test_filtered(oracle, path, prec, tol, n):
    psi0 = oracle.ic_seeds(n, PI4, -0.10, 0.001, 2, 8.0, 0.2, 4)
    ref = oracle.run_filtered(psi0, PI4, -0.3, 0.5, -0.1, -0.5, 0.3, 0.5, 10)
    m = ob.FilteredB200(n, PI4, precision=prec)
    m.initialize(0.5)
    m.set_psi(psi0)
    m.step(10)
    m.sync()
    assert rel_l2(m.get_psi(), ref) <= tol


@pytest.mark.parametrize("prec,tol", [(ob.FP64, 1e-11), (ob.FP32, 1e-5)])
@pytest.mark.parametrize("n", [(64, 64, 64), (128, 64, 32), (512, 16, 32), (32, 16, 1024)])
def test_tungsten(oracle, path, prec, tol, n):
    dx = 1.1107207345395915
    psi0 = np.full((n[2], n[1], n[0]), -0.4)
    origin = [-0.5 * dx * n[a] for a in range(3)]
    psi0 = oracle.ic_seed_inside(psi0, [dx] * 3, origin, 20.0, -0.047, 0.215936)
    p = oracle.TungstenParams.defaults()
    ref = oracle.run_tungsten(psi0, [dx] * 3, p, 1.0, 5)
    m = ob.TungstenB200(n, [dx] * 3, precision=prec)
    m.initialize(1.0)
    m.set_psi(psi0)
    m.step(5)
    m.sync()
    assert rel_l2(m.get_psi(), ref) <= tol


def test_autotune_then_parity(oracle, tmp_path, monkeypatch):
    """The autotuner times every variant, picks one, and the tuned step still
    matches the oracle; a second handle reads the cached choice."""
    monkeypatch.setenv("OPENPFC_GPU_AUTOTUNE_CACHE_DIR", str(tmp_path))
    monkeypatch.delenv("OPENPFC_GPU_AUTOTUNE_MODE", raising=False)
    monkeypatch.delenv("OPFC_Z_VARIANT", raising=False)
    monkeypatch.delenv("OPFC_FP32_COMPUTED_OPERATORS", raising=False)
    n = (64, 64, 64)
    psi0 = oracle.ic_noise(n, -0.285, 0.01, 21)
    ref = oracle.run_plain(psi0, PI4, -0.25, 0.5, 10)
    m = ob.PfcB200(n, PI4, precision=ob.FP32)
    m.initialize(0.5)
    ms = m.autotune()
    assert ms["y.pipelined"] > 0 and ms["y.narrow"] > 0 and ms["z.tables"] > 0 and ms["z.radial"] > 0
    assert ms["z.folded_pingpong"] > 0 and ms["z.direct_folded"] > 0 and ms["z.folded"] > 0
    # FP32 operators computed per mode are candidates only on request
    assert ms["z.computed"] == -1 and ms["z.direct_computed"] == -1 and ms["z.computed_pingpong"] == -1
    assert m.variants()[2] not in (3, 4, 5)
    chosen = m.variants()
    m.set_psi(psi0)
    m.step(10)
    m.sync()
    assert rel_l2(m.get_psi(), ref) <= 1e-5
    assert any(f.name.endswith("_opfc_autotune.json") for f in tmp_path.iterdir())
    m2 = ob.PfcB200(n, PI4, precision=ob.FP32)
    m2.initialize(0.5)
    assert m2.variants() == chosen


def test_transforms(oracle, path):
    n = (128, 64, 512)
    x = np.random.default_rng(2).standard_normal((n[2], n[1], n[0]))
    f = ob.B200Fft(n, precision=ob.FP64)
    X = f.forward(x)
    Xo = oracle.r2c(x)
    assert np.abs(X - Xo).max() <= 1e-12 * np.abs(Xo).max()
    assert np.abs(f.backward(Xo) - oracle.c2r(Xo, n[0])).max() <= 1e-12 * np.abs(x).max()


def test_autotune_fp32_computed_operators_on_request(tmp_path, monkeypatch):
    monkeypatch.setenv("OPENPFC_GPU_AUTOTUNE_CACHE_DIR", str(tmp_path))
    monkeypatch.delenv("OPENPFC_GPU_AUTOTUNE_MODE", raising=False)
    monkeypatch.delenv("OPFC_Z_VARIANT", raising=False)
    monkeypatch.setenv("OPFC_FP32_COMPUTED_OPERATORS", "1")
    m = ob.PfcB200((64, 64, 64), PI4, precision=ob.FP32)
    m.initialize(0.5)
    ms = m.autotune()
    assert ms["z.computed"] > 0 and ms["z.direct_computed"] > 0 and ms["z.computed_pingpong"] > 0


@pytest.mark.parametrize("prec,tol", [(ob.FP64, 1e-11), (ob.FP32, 1e-5)])
@pytest.mark.parametrize("n", [(1024, 32, 32), (32, 1024, 32), (32, 32, 1024)])
def test_filtered_1024_axes(oracle, path, prec, tol, n):
    """Every axis at the measured filtered configuration's length (1024) once,
    with the others short: 1024-point x rows (M = 512), y lines and z lines
    (the z update's W = 4 tiles, its one- and two-stage rings, the (ky, N1 - ky)
    tile order over 1024 rows)."""
    psi0 = oracle.ic_seeds(n, PI4, -0.10, 0.001, 2, 8.0, 0.2, 6)
    ref = oracle.run_filtered(psi0, PI4, -0.3, 0.5, -0.1, -0.5, 0.3, 0.5, 6)
    m = ob.FilteredB200(n, PI4, precision=prec)
    m.initialize(0.5)
    m.set_psi(psi0)
    m.step(6)
    m.sync()
    assert rel_l2(m.get_psi(), ref) <= tol


@pytest.mark.parametrize("off", [("OPENPFC_GPU_AUTOTUNE_DISABLE", "1"), ("OPENPFC_GPU_AUTOTUNE_MODE", "fallback_only"),
                                 ("OPENPFC_GPU_AUTOTUNE_MODE", "cache_only")])
@pytest.mark.parametrize("n", [(64, 64, 64), (256, 48, 256), (512, 16, 1024)])
def test_autotune_without_tuning_keeps_the_defaults(tmp_path, monkeypatch, off, n):
    """Where tuning is switched off, or only an (empty) cache may be read, autotune()
    leaves a handle and an ensemble as initialize() made them."""
    monkeypatch.setenv("OPENPFC_GPU_AUTOTUNE_CACHE_DIR", str(tmp_path))
    monkeypatch.setenv(*off)
    m = ob.FilteredB200(n, PI4, precision=ob.FP32)
    m.initialize(0.5)
    before = m.variants(), m.kernels_per_step()
    m.autotune()
    assert (m.variants(), m.kernels_per_step()) == before
    psi0 = ob.ic_noise((64, 32, 48), -0.285, 0.01, 3)
    got = []
    for tune in (False, True):  # the ensemble's plane kernel rounds differently from its stages
        e = ob.Ensemble([dict(n=(64, 32, 48), dx=PI4, r=-0.2)], precision=ob.FP32)
        e.initialize(0.5)
        if tune:
            e.autotune()
        e.set_psi(0, psi0)
        e.step(5)
        e.sync()
        got.append(e.get_psi(0))
    assert np.array_equal(*got)


def test_autotune_keeps_what_the_environment_forces(tmp_path, monkeypatch):
    """OPFC_PLANE, a forced variant and OPFC_NO_TMA hold after autotune() and against
    a cached choice (64x64x64 FP32 takes the plane kernel: three kernels a step)."""
    monkeypatch.setenv("OPENPFC_GPU_AUTOTUNE_CACHE_DIR", str(tmp_path))
    monkeypatch.delenv("OPENPFC_GPU_AUTOTUNE_MODE", raising=False)

    def kernels(tune, **env):
        with monkeypatch.context() as c:
            for k, v in env.items():
                c.setenv(k, v)
            m = ob.PfcB200((64, 64, 64), PI4, precision=ob.FP32)
            m.initialize(0.5)
            if tune:
                m.autotune()
            return m.kernels_per_step(), m.variants()

    for tune in (True, False):  # False: the cached choices
        assert kernels(tune, OPFC_PLANE="0")[0] == 5
        assert kernels(tune, OPFC_PLANE="1")[0] == 3
        assert kernels(tune, OPFC_X_VARIANT="1")[0] == 5
        assert kernels(tune, OPFC_X_VARIANT="1")[1][1] == 1
        assert kernels(tune, OPFC_Y_VARIANT="2")[1][0] == 2
    f = [f for f in tmp_path.iterdir() if f.name.endswith("_opfc_autotune.json")][0]
    text = f.read_text()
    assert "/xy/" in text
    f.write_text("{\n" + "\n".join(line.replace("[0,", "[1,") if "/xy/" in line else line
                                   for line in text.splitlines()[1:]) + "\n")
    monkeypatch.setenv("OPENPFC_GPU_AUTOTUNE_CACHE_DIR", str(tmp_path) + "/.")  # read the file again
    assert kernels(False)[0] == 3 and kernels(False, OPFC_NO_TMA="1")[0] == 5
