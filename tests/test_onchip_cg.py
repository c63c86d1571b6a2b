"""The on-chip pressure solve (csrc/hf_brick.cu) against the streaming kernel: the same operations in the same order on the
same values, so every field, iteration count and status is equal bit for bit.  Sizes at the edges of its variants: one
tile and less, whole and ragged tiles, blocks of 1, 2, 4, 6, 9 and 15 tiles, p alone on the chip (beyond 15 tiles a block),
the largest that fits and the first that does not."""
import numpy as np
import pytest

from helpers import random_scene_inputs

pytestmark = pytest.mark.gpu


def _scenes(sizes, seed):
    from heatflow_mpm.scene import DeviceScene
    out = []
    for i, n in enumerate(sizes):
        spec, T0, uvw = random_scene_inputs(n, seed=seed + i)
        sc = DeviceScene(spec)
        sc.set_current("T", T0)
        for nm, a in zip("uvw", uvw):
            sc.set_current(nm, a)
        out.append(sc)
    return out


def _equal(a, b):
    for nm in ("T", "u", "v", "w"):
        assert np.array_equal(a.current(nm).cpu().numpy(), b.current(nm).cpu().numpy()), (a.n, nm)
    assert np.array_equal(a.p.cpu().numpy(), b.p.cpu().numpy()), a.n
    sa, sb = a.read_state(), b.read_state()
    assert (sa.pressure_iters, sa.heat_iters, sa.status) == (sb.pressure_iters, sb.heat_iters, sb.status)
    assert (sa.pressure_rr, sa.pressure_bb, sa.rhs_mean) == (sb.pressure_rr, sb.pressure_bb, sb.rhs_mean)


@pytest.mark.parametrize("n", [2, 5, 31, 32, 33, 50, 63, 70, 81, 96, 97, 111, 128, 130, 168, 169])
def test_one_scene_equals_streaming(n):
    from heatflow_mpm.scene import ScenePlan
    (a,), (b,) = _scenes([n], 60), _scenes([n], 60)
    chip, stream = ScenePlan([a]), ScenePlan([b], streaming_cg=True)
    for plan in (chip, stream):
        plan.prepare_statics()
        for _ in range(2):
            plan.substep(2e-3)
    _equal(a, b)


@pytest.mark.parametrize("sizes", [(20, 33, 47), (96, 96, 64, 64, 48, 40, 33, 32) * 2, (128, 24, 128, 57), (136, 40, 88)],
                         ids=["side by side", "in turn", "large first", "p alone"])
def test_batch_equals_streaming(sizes):
    """Teams that share the blocks at the same time and one after another, over several launches of one plan."""
    from heatflow_mpm.scene import ScenePlan
    chip, stream = _scenes(sizes, 90), _scenes(sizes, 90)
    for plan in (ScenePlan(chip), ScenePlan(stream, streaming_cg=True)):
        plan.prepare_statics()
        for _ in range(2):
            plan.substep(2e-3)
    for a, b in zip(chip, stream):
        _equal(a, b)


def test_launch_number_wraps():
    """The tags keep 12 bits of the launch number.  A heat solve of one iteration, solves of none up to the wrap, then one
    that iterates again from another state, with the first one's tags: it equals the streaming kernel's, bit for bit (no
    block takes a sum that the first launch left behind)."""
    import torch
    from heatflow_mpm.scene import ScenePlan
    dt = 2e-3
    (a,), (b,) = _scenes([24], 60), _scenes([24], 60)
    chip, stream = ScenePlan([a]), ScenePlan([b], streaming_cg=True)
    rng = np.random.default_rng(4)
    first, last = ((25.0 + rng.uniform(-c, c, (24, 24, 24))).astype(np.float32) for c in (2.0, 9.0))
    for plan, sc in ((chip, a), (stream, b)):
        plan.prepare_statics()
        nxt = sc.T[sc.parity() ^ 1]
        for start in (first, last):
            nxt.copy_(torch.as_tensor(start))
            sc.hrhs.copy_(torch.as_tensor(start))
            plan.heat_solve(dt)
            iters = sc.read_state().heat_iters
            assert iters == 1 if start is first else iters >= 1
            if start is first and plan is chip:
                for _ in range(4095):
                    plan.heat_solve(dt)
                assert sc.read_state().heat_iters == 0
        sc.result = nxt.cpu().numpy()
    assert np.array_equal(a.result, b.result)
    assert a.read_state().heat_rr == b.read_state().heat_rr and a.read_state().status == 0


def test_step_numbers_wrap():
    """The tags keep 10 bits of the step: more than 1024 iterations (two steps and one halo exchange each), forced by face
    fractions over six decades."""
    import torch
    from heatflow_mpm.scene import ScenePlan
    (a,), (b,) = _scenes([32], 60), _scenes([32], 60)
    for sc in (a, b):
        sc.spec.cg_max_iter, sc.spec.cg_tol = 1200, 1e-30
    rng = np.random.default_rng(6)
    weights = [torch.as_tensor((10.0 ** rng.uniform(-6, 0, s.shape)).astype(np.float32)) for s in (a.ax, a.ay, a.az)]
    for sc, plan in ((a, ScenePlan([a])), (b, ScenePlan([b], streaming_cg=True))):
        plan.prepare_statics()
        for dst, w in zip((sc.ax, sc.ay, sc.az), weights):
            dst.copy_(w)
        for dst, w in ((sc.ayc, sc.ay[:, :-1]), (sc.azc, sc.az[:, :, :-1])):
            dst.copy_(w)
        plan.substep(2e-3)
    assert a.read_state().pressure_iters == 1200
    _equal(a, b)


def test_quotient_is_the_operators():
    """The division that gives alpha and beta against numpy's, bit for bit: significands at random, divisors with every bit
    set and their neighbours, quotients beside the midpoint of two doubles, and any bit patterns at all (zeros, subnormals,
    infinities and NaNs among them)."""
    import torch
    from heatflow_mpm import _lib
    L = _lib.load()
    rng = np.random.default_rng(8)
    N = 1 << 20
    man = lambda: 1.0 + rng.integers(0, 1 << 52, N) * 2.0 ** -52
    exp = lambda: np.ldexp(rng.choice([-1.0, 1.0], N), rng.integers(-99, 100, N))
    ulps = lambda k: rng.integers(0, k, N) * 2.0 ** -52
    pairs = [(man() * exp(), man() * exp()), ((1.0 + ulps(64)) * exp(), (2.0 - 2.0 ** -52 - ulps(64)) * exp()),
             ((2.0 - 2.0 ** -52 - ulps(1024)) * exp(), (1.0 + ulps(1024)) * exp())]
    b = man()
    mid = man().astype(np.longdouble) + np.longdouble(2.0) ** -53
    pairs.append(((mid * b.astype(np.longdouble)).astype(np.float64), b))
    anything = rng.integers(-2 ** 63, 2 ** 63 - 1, (2, N), dtype=np.int64).view(np.float64)
    pairs.append((anything[0], anything[1]))
    special = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, 2.0 ** -100, 2.0 ** 100, np.nextafter(2.0 ** 100, 4e30), 1.0, -3.0])
    pairs.append(tuple(x.ravel() for x in np.meshgrid(special, special)))
    for a, b in pairs:
        dev = [torch.as_tensor(np.ascontiguousarray(v), device="cuda") for v in (a, b)]
        out = torch.empty_like(dev[0])
        _lib.check(L.hf_k_quotient(out.numel(), dev[0].data_ptr(), dev[1].data_ptr(), out.data_ptr(),
                                   torch.cuda.current_stream().cuda_stream), "hf_k_quotient")
        with np.errstate(all="ignore"):
            want = a / b
        got = out.cpu().numpy()
        bad = (got.view(np.int64) != want.view(np.int64)) & ~(np.isnan(got) & np.isnan(want))
        assert not bad.any(), (int(bad.sum()), a[bad][0].hex(), b[bad][0].hex(), got[bad][0].hex(), want[bad][0].hex())


@pytest.mark.parametrize("sizes,blocks,lanes", [((70,), 3, 0), ((70,), 0, 0), ((97, 33, 150), 2, 1), ((50, 49, 53, 54), 8, 2)], ids=str)
def test_streaming_sums_by_units(sizes, blocks, lanes):
    """The streaming kernel's scene sums, whose partials are spread by unit, for blocks of more tiles than keep their places (162
    and 2072 of them), units of one tile and of one and two, and scenes that share a lane: the on-chip solve's bits."""
    from heatflow_mpm.scene import ScenePlan
    chip, stream = _scenes(sizes, 75), _scenes(sizes, 75)
    for plan in (ScenePlan(chip), ScenePlan(stream, streaming_cg=True, persistent_blocks=blocks, lanes=lanes)):
        plan.prepare_statics()
        plan.substep(2e-3)
    for a, b in zip(chip, stream):
        _equal(a, b)
