"""Learned distance surrogate on the GPU.

* Forward pass (tcgen05 and mma.sync engines) and gradients of the BF16
  tensor-core kernels against the FP64
  oracle that rounds to BF16 where the kernels store BF16 (the remaining
  differences: FP32 accumulation order, the hardware tanh/sin/cos, BF16
  rounding-boundary flips; inference takes its sigmoid from an f16x2 tanh).
  Tolerances: forward |dy| <= 3e-3 * (max|y| + 0.1) for 99% of points;
  per parameter block ||g - g_ref|| <= 2e-2 ||g_ref||.
* Training on the GPU lowers the asymmetric loss by 10x and keeps
  overestimates rare.
* The skip march gives the same hits as the plain march: hit/miss
  agreement >= 99.5% and hit-distance error versus the FP64 oracle within
  1.5x the plain march's own 99th percentile (both within 5e-5 (1 + t)); it
  reports the exact DE evaluations with the trained network, without it
  (the same march with the model's box only) and without the skip pass, and
  checks that the network lowers the exact evaluations below the box-only
  march.
"""
import numpy as np
import pytest

import oracle
from fractalpathtracer_gb300 import native_ext as nx
from fractalpathtracer_gb300 import scenes

pytestmark = pytest.mark.gpu

BULB_BOX = scenes.SURROGATE_BOXES["mandelbulb"]


def _points(n, seed):
    rng = np.random.default_rng(seed)
    p = np.zeros((n, 4), np.float32)
    p[:, :3] = rng.uniform(-1.2, 1.2, (n, 3))
    p[:, 3] = rng.uniform(-0.05, 0.6, n)
    return p


@pytest.fixture(scope="module")
def blank_model(native):
    cfg, ext = scenes.mandelbulb_primary(8, 8)
    mc = nx.mlp_config(*BULB_BOX, points=0, steps=0)
    h, _ = nx.mlp_create(cfg, ext, mc)
    yield h
    nx.mlp_destroy(h)


@pytest.fixture
def engine(request):
    nx.set_network_engine(request.param)
    yield request.param
    nx.set_network_engine(nx.NET_TCGEN05)


ENGINES = [pytest.param(nx.NET_TCGEN05, id="tcgen05"), pytest.param(nx.NET_MMA_SYNC, id="mma_sync")]


@pytest.mark.parametrize("engine", ENGINES, indirect=True)
def test_forward_matches_oracle(blank_model, engine):
    params = scenes.random_mlp_params(11)
    nx.mlp_set_params(blank_model, params)
    back = nx.mlp_get_params(blank_model)
    assert np.array_equal(back, params)
    pts = _points(4096 + 77, 5)   # a ragged last tile
    y = nx.mlp_predict(blank_model, pts).astype(np.float64)
    ref = oracle.mlp_forward(params, *BULB_BOX, pts, emulate_bf16=True)
    err = np.abs(y - ref)
    scale = np.abs(ref).max() + 0.1
    print(f"forward ({engine}): max|y| {np.abs(ref).max():.3f} p99 err {np.percentile(err, 99):.2e} max err {err.max():.2e}")
    assert np.percentile(err, 99) <= 3e-3 * scale
    assert err.max() <= 1.5e-2 * scale


def test_engines_agree(blank_model):
    """tcgen05 and mma.sync compute the same network; only FP32 summation order differs (and BF16 rounding flips
    of activations that it moves across a rounding boundary)."""
    params = scenes.random_mlp_params(12)
    nx.mlp_set_params(blank_model, params)
    pts = _points(1 << 16, 6)
    try:
        nx.set_network_engine(nx.NET_MMA_SYNC)
        y_mma = nx.mlp_predict(blank_model, pts).astype(np.float64)
    finally:
        nx.set_network_engine(nx.NET_TCGEN05)
    y_tc = nx.mlp_predict(blank_model, pts).astype(np.float64)
    d = np.abs(y_tc - y_mma)
    scale = np.abs(y_mma).max() + 0.1
    print(f"tcgen05 vs mma.sync: identical {np.mean(d == 0):.4f} p99 {np.percentile(d, 99):.2e} max {d.max():.2e}")
    assert np.percentile(d, 99) <= 1e-3 * scale
    assert d.max() <= 1e-2 * scale


@pytest.mark.parametrize("engine", ENGINES, indirect=True)
def test_gradients_match_oracle(blank_model, engine):
    """Gradients and loss of one pass against the FP64 oracle, with the training's forward/backward on either
    engine (tcgen05 by default, mma.sync); the weight gradients run on tcgen05 in both."""
    params = scenes.random_mlp_params(12)
    nx.mlp_set_params(blank_model, params)
    pts = _points(1000, 6)   # not a multiple of the 128-row block: exercises the ragged tail
    g, loss = nx.mlp_gradients(blank_model, pts, 10.0)
    g_ref, loss_ref = oracle.mlp_gradients(params, *BULB_BOX, pts, 10.0, emulate_bf16=True)
    assert abs(loss - loss_ref) <= 5e-3 * loss_ref
    blocks = {"W0": (0, 7168), "b0": (7168, 7232), "W1": (7232, 11328), "b1": (11328, 11392), "W2": (11392, 15488),
              "b2": (15488, 15552), "W3": (15552, 19648), "b3": (19648, 19712), "W4": (19712, 19776), "b4": (19776, 19777)}
    for name, (a, b) in blocks.items():
        d = np.linalg.norm(g[a:b] - g_ref[a:b])
        r = np.linalg.norm(g_ref[a:b])
        print(f"{name}: |g| {r:.3e} rel err {d / max(r, 1e-30):.2e}")
        assert d <= 2e-2 * r + 1e-7, name
    pad = g[:7168].reshape(64, 112)[:, 99:]
    assert np.abs(pad).max() < 1e-3 * np.abs(g[:7168]).max()   # padding columns carry no real gradient


@pytest.mark.parametrize("rows", [1, 8, 63, 65, 128, 129, 255, 257, 449])
def test_gradient_tile_edges(blank_model, rows):
    """Batches that end inside an 8-row block, a 64-row tile, a 128-row CTA and a 256-row chunk, against the oracle
    (the tolerance of test_gradients_match_oracle, over the whole gradient)."""
    params = scenes.random_mlp_params(14)
    nx.mlp_set_params(blank_model, params)
    pts = _points(rows, 9)
    g, loss = nx.mlp_gradients(blank_model, pts, 10.0)
    g_ref, loss_ref = oracle.mlp_gradients(params, *BULB_BOX, pts, 10.0, emulate_bf16=True)
    assert abs(loss - loss_ref) <= 2e-2 * loss_ref
    assert np.linalg.norm(g - g_ref) <= 2e-2 * np.linalg.norm(g_ref) + 1e-7


def test_gradients_are_deterministic(blank_model):
    """The weight and bias gradients come from tcgen05 MMAs per 512-row chunk and a reduction in chunk order, the
    output layer and the loss from per-warp sums added in warp order: no floating-point atomics, so the same batch
    gives the same bits (here 20000 rows: 40 chunks, the last one ragged)."""
    params = scenes.random_mlp_params(13)
    nx.mlp_set_params(blank_model, params)
    pts = _points(20000, 8)
    g1, l1 = nx.mlp_gradients(blank_model, pts, 10.0)
    g2, l2 = nx.mlp_gradients(blank_model, pts, 10.0)
    assert np.array_equal(g1, g2) and l1 == l2
    g_ref, _ = oracle.mlp_gradients(params, *BULB_BOX, pts, 10.0, emulate_bf16=True)
    assert np.linalg.norm(g1 - g_ref) <= 2e-2 * np.linalg.norm(g_ref)


def test_training_is_deterministic(native):
    """Two trainings from the same seed on uniformly sampled points end with the same parameters, bit for bit.
    (Near-surface points are appended by warp-aggregated atomics, so the sample set of a run with near_fraction > 0
    can differ in the points kept from the last rejection round.)"""
    cfg, ext = scenes.mandelbulb_primary(8, 8)
    mc = nx.mlp_config(*BULB_BOX, points=1 << 18, near_fraction=0.0, steps=60, batch=4096, lr=2e-3, seed=5)
    params = []
    for _ in range(2):
        h, _ = nx.mlp_create(cfg, ext, mc)
        try:
            params.append(nx.mlp_get_params(h))
        finally:
            nx.mlp_destroy(h)
    assert np.array_equal(params[0], params[1])


def _pcg(v):
    v = np.asarray(v, np.uint32)
    state = v * np.uint32(747796405) + np.uint32(2891336453)
    word = ((state >> ((state >> np.uint32(28)) + np.uint32(4))) ^ state) * np.uint32(277803737)
    return (word >> np.uint32(22)) ^ word


@pytest.mark.parametrize("engine", ENGINES, indirect=True)
@pytest.mark.parametrize("rows,steps", [(64, 1), (333, 2), (4096 + 77, 3)])
def test_training_steps_match_adam_on_the_host(native, blank_model, engine, rows, steps):
    """One to three training steps, ragged batches among them, against Adam in FP32 on the host with the gradients of
    fpt_cuda_mlp_gradients at the same rows.  A parameter moves by at most about lr a step; the host's separately rounded
    operations and the few BF16 weights that they flip change a step by less than 1e-5 (0.5% of lr) for nearly all.  The
    BF16 weights of the trained model are those of its parameters, and the padding columns of W0 stay zero."""
    cfg, ext = scenes.mandelbulb_primary(8, 8)
    points, seed, lr0 = 2048, 21, 2e-3
    mc = nx.mlp_config(*BULB_BOX, points=points, near_fraction=0.0, steps=steps, batch=rows, lr=lr0, seed=seed)
    h, _ = nx.mlp_create(cfg, ext, mc)
    try:
        trained = nx.mlp_get_params(h)
        probe = _points(1000, 4)
        predicted = nx.mlp_predict(h, probe)
    finally:
        nx.mlp_destroy(h)
    h, _ = nx.mlp_create(cfg, ext, nx.mlp_config(*BULB_BOX, points=0, steps=0, seed=seed))
    try:
        p = nx.mlp_get_params(h)
    finally:
        nx.mlp_destroy(h)
    index = np.arange(points, dtype=np.uint32)
    hashed = _pcg(np.uint32(seed) ^ _pcg(index))
    data = np.zeros((points, 4), np.float32)
    lo, hi = (np.asarray(b, np.float64) for b in BULB_BOX)
    for k in range(3):
        data[:, k] = lo[k] + (hi[k] - lo[k]) * ((_pcg(hashed + np.uint32(k)) >> np.uint32(8)) / 16777216.0)
    data[:, 3] = native.sample_distance(cfg, ext, data)[:, 0]
    f = np.float32
    m, v = np.zeros_like(p), np.zeros_like(p)
    for s in range(steps):
        nx.mlp_set_params(blank_model, p)
        pick = _pcg(np.uint32(seed + 7919 * s) ^ _pcg(np.arange(rows, dtype=np.uint32))) % np.uint32(points)
        g, _ = nx.mlp_gradients(blank_model, data[pick], 10.0)
        g[:7168].reshape(64, 112)[:, 99:] = 0.0
        lr = f(max(lr0 * 0.5 * (1.0 + np.cos(np.pi * s / steps)), lr0 * 0.02))
        m = f(0.9) * m + f(0.1) * g
        v = f(0.999) * v + f(0.001) * g * g
        p = p - lr * (m / f(1.0 - 0.9 ** (s + 1))) / (np.sqrt(v / f(1.0 - 0.999 ** (s + 1))) + f(1e-8))
    off = np.abs(trained - p)
    print(f"{rows} rows, {steps} steps: max {off.max():.2e} p99.5 {np.percentile(off, 99.5):.2e}")
    assert np.percentile(off, 99.5) <= 1e-5
    assert off.max() <= 2 * lr0 * steps
    assert not trained[:7168].reshape(64, 112)[:, 99:].any()
    nx.mlp_set_params(blank_model, trained)
    assert np.array_equal(nx.mlp_predict(blank_model, probe), predicted)


@pytest.fixture(scope="module")
def trained_bulb(native):
    cfg, ext = scenes.mandelbulb_primary(8, 8)
    mc = nx.mlp_config(*BULB_BOX, points=1 << 20, steps=800, batch=8192, lr=2e-3, seed=3)
    h, stats = nx.mlp_create(cfg, ext, mc)
    print("training:", stats)
    yield h, stats
    nx.mlp_destroy(h)


def test_training_reduces_loss_and_underestimates(trained_bulb, native):
    h, stats = trained_bulb
    assert stats["near_points"] == (1 << 19)
    assert stats["loss_last"] < 0.1 * stats["loss_first"], stats
    cfg, ext = scenes.mandelbulb_primary(8, 8)
    rng = np.random.default_rng(9)
    pts = np.zeros((65536, 4), np.float32)
    pts[:, :3] = rng.uniform(-1.25, 1.25, (65536, 3))
    exact = native.sample_distance(cfg, ext, pts)[:, 0].astype(np.float64)
    pred = nx.mlp_predict(h, pts).astype(np.float64)
    err = pred - exact
    over = (err > 0.02).mean()
    under = (err < -0.02).mean()
    print(f"held-out: mean |err| {np.abs(err).mean():.4f} over>0.02 {over:.4f} under<-0.02 {under:.4f}")
    assert np.abs(err).mean() < 0.05
    assert over < under + 0.01


def _hits(native, cfg, ext):
    hits, ms = native.trace_primary(cfg, ext)
    return hits, ms


@pytest.mark.parametrize("engine", ENGINES, indirect=True)
def test_skip_march_keeps_hits(trained_bulb, native, engine):
    h, _ = trained_bulb
    cfg, ext = scenes.mandelbulb_primary(320, 240)
    plain, _ = _hits(native, cfg, ext)
    ref = oracle.trace_primary(cfg, ext, fp64=True)

    def run(model, mode=1):
        e = scenes.mandelbulb_primary(320, 240)[1]
        e.surrogate = mode
        e.surrogate_model = model
        hits, _ = _hits(native, cfg, e)
        return hits, nx.skip_stats()

    skip, st = run(h)
    # the same march without the network: the model's box only
    nonet, st0 = run(h, mode=2)
    hit_r = ref[..., 5] > 0
    rows = []
    for name, g in (("plain", plain), ("skip", skip), ("no-network", nonet)):
        hit_g = g["hit"] > 0
        both = hit_g & hit_r
        derr = np.abs(g["distance"][both] - ref[..., 0][both]) / (1 + ref[..., 0][both])
        rows.append((name, (hit_g == hit_r).mean(), np.percentile(derr, 99), int(g["steps"].astype(np.int64).sum())))
    for r in rows:
        print("%-10s agree %.5f p99 dist err %.2e exact evals %d" % r)
    print("skip stats:", st)
    print("no-network stats:", st0)
    (_, a0, e0, n0), (_, a1, e1, n1), (_, a2, e2, n2) = rows
    assert a1 >= 0.995 and a2 >= 0.995
    assert e1 <= 5e-5 and e1 <= 1.5 * e0 + 1e-6
    assert e2 <= 5e-5
    assert st["accepted"] > 0 and st["rows"] > 0
    assert st0["rows"] == 0 and st0["accepted"] == 0
    assert n1 < n2 < n0   # network < box only < plain
    agree = ((skip["hit"] > 0) == (plain["hit"] > 0)).mean()
    assert agree >= 0.995


def test_skip_render_matches_plain(trained_bulb, native):
    """Path tracing with the skip pass in front of every march pass: same seed, same image as the plain march
    within sampling noise of paths whose hit points moved by less than the hit threshold."""
    import ctypes
    h, _ = trained_bulb
    b = scenes.mandelbulb_path(256, 144, 8, 4)
    _, rgba_p, _ = native.cuda_render(b.cfg, b.ext, linear=False)
    e = type(b.ext)()
    ctypes.memmove(ctypes.byref(e), ctypes.byref(b.ext), ctypes.sizeof(b.ext))
    e.surrogate = 1
    e.surrogate_model = h
    _, rgba_s, _ = native.cuda_render(b.cfg, e, linear=False)
    st = nx.skip_stats()
    m = oracle.image_metrics(rgba_p, rgba_s)
    print("skip vs plain render:", m, st)
    assert st["accepted"] > 0 and st["escaped"] > 0
    assert m["mae"] <= 2.0 and m["lf_ssim"] >= 0.98, m


def test_mandelbox_skip(native):
    """The learned skip on the second surrogate scene, the scale -1.5 Mandelbox: a model trained on its own
    DE; primary-ray hits equal to the plain march's and a render equal to the plain render within noise."""
    import ctypes
    b = scenes.mandelbox_path(256, 144, 8, 4)
    lo, hi = scenes.SURROGATE_BOXES["mandelbox"]
    h, stats = nx.mlp_create(b.cfg, b.ext, nx.mlp_config(lo, hi, points=1 << 20, steps=800, batch=8192, lr=2e-3, seed=4))
    try:
        assert stats["loss_last"] < 0.1 * stats["loss_first"], stats
        e = type(b.ext)()
        ctypes.memmove(ctypes.byref(e), ctypes.byref(b.ext), ctypes.sizeof(b.ext))
        e.surrogate, e.surrogate_model = 1, h
        hp, _ = native.trace_primary(b.cfg, b.ext)
        hs, _ = native.trace_primary(b.cfg, e)
        st_primary = nx.skip_stats()
        agree = ((hp["hit"] > 0) == (hs["hit"] > 0)).mean()
        both = (hp["hit"] > 0) & (hs["hit"] > 0)
        dt = np.abs(hp["distance"][both].astype(np.float64) - hs["distance"][both]) / (1.0 + hp["distance"][both])
        print(f"mandelbox primary: agree {agree:.5f} p99 rel dist delta {np.percentile(dt, 99):.2e}", st_primary)
        assert agree >= 0.995 and np.percentile(dt, 99) <= 5e-5
        assert st_primary["accepted"] > 0
        _, rgba_p, _ = native.cuda_render(b.cfg, b.ext, linear=False)
        _, rgba_s, _ = native.cuda_render(b.cfg, e, linear=False)
        m = oracle.image_metrics(rgba_p, rgba_s)
        print("mandelbox skip vs plain render:", m, nx.skip_stats())
        assert m["mae"] <= 2.0 and m["lf_ssim"] >= 0.98, m
    finally:
        nx.mlp_destroy(h)


def test_bounded_mbarrier_wait(blank_model):
    """The tensor-core kernels' mbarrier waits are bounded: a wait that nothing completes runs out after its
    limit and reports it, the kernel frees its tensor memory, and tcgen05 kernels run normally afterwards."""
    r = nx.bounded_wait_check()
    print(r)
    assert r["arrived"] == 1 and r["arrived_ns"] < 5_000_000
    assert r["not_arrived"] == 2 and 20_000_000 <= r["not_arrived_ns"] < 1_000_000_000
    nx.set_network_engine(nx.NET_TCGEN05)
    y = nx.mlp_predict(blank_model, _points(256, 7))
    assert np.isfinite(y).all()


@pytest.mark.parametrize("scene", ["mandelbulb", "mandelbox"])
def test_perfect_proposal_bound(native, scene):
    """fpt_cuda_certified_steps: in total a perfect proposal needs no more evaluations than the plain march for
    camera, shadow and bounce rays; the ratio is the most any network can save under the skip's certificate.  Per
    ray it is not monotone (measured: 1.4% of the Mandelbulb's and 4.4% of the Mandelbox's camera rays take more):
    a longer certified step leaves the ray at another position, from which the remaining march can take longer."""
    b = scenes.mandelbulb_path(480, 270, 1) if scene == "mandelbulb" else scenes.mandelbox_path(480, 270, 1)
    c = native.certified_steps(b.cfg, b.ext, list(b.ext.sun_direction), stride=2, margin=0.1).astype(np.int64)
    bound = nx.certified_step_bound(b.cfg, b.ext, list(b.ext.sun_direction), stride=2, margin=0.0)
    print(scene, bound)
    for k in range(3):
        plain, cert = c[:, 2 * k], c[:, 2 * k + 1]
        has = plain > 0
        assert has.sum() > 100
        assert cert[has].sum() <= plain[has].sum()
        assert np.mean(cert[has] <= plain[has] + 1) > 0.9
    for k in ("camera", "shadow", "bounce"):
        assert bound[k]["ratio"] >= 1.0
