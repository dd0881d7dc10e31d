"""Batch distance samples on the GPU vs the FP64 oracle.

Gate of the reference's mandel-parity command (src/main.rs:3297,
3356-3361): |d_gpu - d_fp64| <= 5e-5 * (1 + |d_fp64|), p99 within the
gate, outlier fraction <= 2e-4 (here 1e-3 for the FP32 algebraic form of
the power-8 step against the FP64 trigonometric form).
"""
import numpy as np
import pytest

import oracle
from fractalpathtracer_gb300 import ffi, scenes

pytestmark = pytest.mark.gpu


def pts(n, lo, hi, seed=11):
    p = np.random.default_rng(seed).uniform(lo, hi, (n, 4)).astype(np.float32)
    p[:, 3] = 0
    return p


def _gate(d_gpu, d_ref, outliers=1e-3):
    err = np.abs(d_gpu - d_ref) / (1 + np.abs(d_ref))
    assert np.percentile(err, 99) <= 5e-5, np.percentile(err, 99)
    assert np.mean(err > 5e-5) <= outliers, np.mean(err > 5e-5)


def test_mandelbulb_field(native):
    cfg, ext = scenes.mandelbulb_primary(8, 8)
    p = pts(1 << 16, -1.5, 1.5)
    g = native.sample_distance(cfg, ext, p)
    r = oracle.sample_distance(cfg, ext, p, fp64=True)
    _gate(g[:, 0], r[:, 0])
    assert np.mean(g[:, 3] == r[:, 3]) > 0.999   # iteration counts


def test_mandelbox_field(native):
    b = scenes.mandelbox_path(8, 8, 1)
    p = pts(1 << 16, -4, 4)
    g = native.sample_distance(b.cfg, b.ext, p)
    r = oracle.sample_distance(b.cfg, b.ext, p, fp64=True)
    _gate(g[:, 0], r[:, 0])


def test_reference_ifs_field_sample(native):
    """fpt_mandelbulber_sample_field with the built-in Kaleidoscopic IFS (shaders/Shaders.metal:901-954)."""
    cfg = ffi.default_config()
    cfg.sdf_id = ffi.SDF_MANDELBULBER
    s = cfg.set_values
    s[0], s[1], s[2], s[3] = 1.0, 12.0, 10.0, 2.0
    s[4], s[5] = 7.0, 7.0                      # abs xyz, three fold planes
    s[6], s[7], s[8] = 1.0, 1.0, 1.0
    dirs = [(1, -1, 0), (0, 1, -1), (1, 0, -1)]
    for k, d in enumerate(dirs):
        n = np.array(d, float) / np.linalg.norm(d)
        s[12 + 3 * k:15 + 3 * k] = list(n)
    p = pts(1 << 15, -2, 2)
    g = native.sample_field(cfg, p)
    r = oracle.field_sample(cfg, None, p, fp64=True)
    _gate(g[:, 0], r[:, 0])
    assert np.mean(g[:, 3] == r[:, 3]) > 0.999


def test_analytic_gradient_matches_fp64(native):
    cfg, ext = scenes.mandelbulb_primary(8, 8)
    p = pts(4096, -1.3, 1.3)
    _, gg = native.sample_distance(cfg, ext, p, gradients=True)
    _, gr = oracle.sample_distance(cfg, ext, p, fp64=True, gradients=True)
    ng = np.linalg.norm(gg, axis=1)
    nr = np.linalg.norm(gr, axis=1)
    ok = (nr > 1e-6) & np.isfinite(ng)
    cosang = (gg[ok] * gr[ok]).sum(1) / (ng[ok] * nr[ok])
    assert np.percentile(np.degrees(np.arccos(np.clip(cosang, -1, 1))), 99) < 0.5


# Mandelbulbs of power 2.29, 10.6, 2.89, 5.24, 7.93; Mandelboxes; hybrids of 5, 12 and 16 iterations.
@pytest.mark.parametrize("k", [11, 14, 21, 27, 30, 1, 9, 12, 0, 3, 4])
def test_batch_scene_fields(native, k):
    """The formulas of the batched workload against the FP64 oracle: Mandelbulbs of non-integer power (the
    trigonometric step of orbit.rs:766-778), Mandelboxes of other scales, the bulb / Menger hybrid, with
    4-16 iterations (scene k of scenes.batch_scene)."""
    b = scenes.batch_scene(k)
    p = pts(1 << 15, -1.6 if b.ext.formula != ffi.FORMULA_MANDELBOX else -4.0,
            1.6 if b.ext.formula != ffi.FORMULA_MANDELBOX else 4.0, seed=20 + k)
    g = native.sample_distance(b.cfg, b.ext, p)
    r = oracle.sample_distance(b.cfg, b.ext, p, fp64=True)
    print(k, b.ext.formula, b.ext.power, b.ext.iterations,
          np.percentile(np.abs(g[:, 0] - r[:, 0]) / (1 + np.abs(r[:, 0])), 99))
    _gate(g[:, 0], r[:, 0], outliers=5e-3)
    assert np.mean(g[:, 3] == r[:, 3]) > 0.99   # iteration counts


def test_mandelbulb_power2_triplex_field(native):
    """Mandelbulber formula 3, the quadratic triplex of orbit.rs:752-764 (known answer pinned on the CPU at
    orbit.rs:1866-1874), marched as a scene: GPU field and analytic gradient against the FP64 oracle."""
    cfg, ext = scenes.mandelbulb_primary(8, 8)
    ext.formula = ffi.FORMULA_MANDELBULB_POWER2
    ext.iterations = 10
    ext.bailout = 4.0
    p = pts(1 << 16, -1.6, 1.6, seed=5)
    g, gg = native.sample_distance(cfg, ext, p, gradients=True)
    r, gr = oracle.sample_distance(cfg, ext, p, fp64=True, gradients=True)
    _gate(g[:, 0], r[:, 0])
    assert np.mean(g[:, 3] == r[:, 3]) > 0.999
    ng, nr = np.linalg.norm(gg, axis=1), np.linalg.norm(gr, axis=1)
    ok = (nr > 1e-6) & np.isfinite(ng) & (np.abs(r[:, 0]) > 1e-3)
    cosang = (gg[ok] * gr[ok]).sum(1) / (ng[ok] * nr[ok])
    assert np.percentile(np.degrees(np.arccos(np.clip(cosang, -1, 1))), 99) < 0.5


def _bulb8_f32(points, iterations, bailout):
    """The algebraic power-8 orbit in FP32: (rho + i z)^8 times ((x + i y) / rho)^8, as the kernels compute it."""
    f = np.float32
    out = np.zeros(len(points))
    for k, (px, py, pz) in enumerate(points[:, [0, 2, 1]].astype(f)):   # the field's axes: world x, z, y
        x, y, z, dr = px, py, pz, f(1)
        r = np.sqrt(x * x + y * y + z * z)
        for _ in range(iterations):
            rho = np.sqrt(x * x + y * y)
            w, e = np.array([rho, z], f), np.array([x / rho, y / rho] if rho > 0 else [1, 0], f)
            for _ in range(3):
                w = np.array([w[0] * w[0] - w[1] * w[1], 2 * w[0] * w[1]], f)
                e = np.array([e[0] * e[0] - e[1] * e[1], 2 * e[0] * e[1]], f)
            dr = r ** f(7) * dr * f(8) + f(1)
            x, y, z = w[0] * e[0] + px, w[0] * e[1] + py, w[1] + pz
            r = np.sqrt(x * x + y * y + z * z)
            if r > bailout:
                break
        out[k] = 0.5 * r * np.log(r) / dr if r > 1 else 0.0
    return out


@pytest.mark.parametrize("iterations,bailout", [(1, 2.0), (2, 1.0), (8, 2.0), (5, 50.0)])
def test_mandelbulb8_step_edges(native, iterations, bailout):
    """The power-8 step's branches: the polar axis (x = y = 0), coordinate planes, the origin, points whose squares
    are denormal or zero, and orbits that stop at the first iteration or never escape."""
    cfg, ext = scenes.mandelbulb_primary(8, 8)
    ext.iterations, ext.bailout = iterations, bailout
    p = pts(4096, -1.4, 1.4, seed=3)
    p[:512, 0] = 0.0
    p[256:768, 2] = 0.0          # the field's y: with the first lines, points of the polar axis
    p[768:1024, 1] = 0.0
    p[1024:1536, :3] *= np.float32(1e-19)
    p[1536:1792, 0] *= np.float32(1e-22)
    p[1536:1792, 2] *= np.float32(1e-22)
    p[1792, :3] = 0.0
    g = native.sample_distance(cfg, ext, p)
    r = oracle.sample_distance(cfg, ext, p, fp64=True)
    flat = slice(1536, 1792)     # x^2 + y^2 is denormal: FP32 has no angle left there, so FP32 is the reference
    r[flat, 0] = _bulb8_f32(p[flat], iterations, bailout)
    _gate(g[:, 0], r[:, 0], outliers=5e-3)
    assert np.mean(g[:, 3] == r[:, 3]) > 0.995


@pytest.mark.parametrize("scale", [1.0, 2.5])
@pytest.mark.parametrize("box", [False, True])
def test_world_scale(native, box, scale):
    """The field's world scale: 1, where nothing is divided, and another."""
    if box:
        b = scenes.mandelbox_path(8, 8, 1)
        cfg, ext, reach = b.cfg, b.ext, 4.0
    else:
        cfg, ext = scenes.mandelbulb_primary(8, 8)
        reach = 1.5
    cfg.set_values[0] = scale
    p = pts(1 << 13, -reach * scale, reach * scale, seed=17)
    g = native.sample_distance(cfg, ext, p)
    r = oracle.sample_distance(cfg, ext, p, fp64=True)
    _gate(g[:, 0], r[:, 0])
    assert np.mean(g[:, 3] == r[:, 3]) > 0.995


LARGEST = float(np.finfo(np.float32).max)


@pytest.mark.parametrize("route", ["bailout", "set_values"])
@pytest.mark.parametrize("iterations", [1, 2, 3, 8, 40])
def test_mandelbulb8_without_bailout(native, iterations, route):
    """Power-8 orbits that end where FP32 overflows: an infinite bailout radius rolls the last step back like the largest
    finite one does, bit for bit.  The FP32 oracle is the reference (FP64 overflows some iterations later)."""
    p = pts(4096, -1.4, 1.4, seed=3)
    p[:512, :3] *= np.float32(100.0)     # over at the first or second step
    out = []
    for bailout in (np.inf, LARGEST):
        cfg, ext = scenes.mandelbulb_primary(8, 8)
        ext.iterations = iterations
        ext.bailout = bailout if route == "bailout" else 0.0
        cfg.set_values[2] = bailout
        out.append(native.sample_distance(cfg, ext, p))
        r = oracle.sample_distance(cfg, ext, p, fp64=False)
    assert np.isfinite(out[0]).all(axis=0)[[0, 1, 3]].all()   # the derivative of a rolled-back step may overflow
    assert np.array_equal(out[0], out[1], equal_nan=True)
    _gate(out[0][:, 0], r[:, 0], outliers=5e-3)
    assert np.mean(out[0][:, 3] == r[:, 3]) > 0.995
