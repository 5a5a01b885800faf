"""Launches of few rays take one block per SM, and the shape changes no bit of
a render: the kernels whose geodesic is FP64 (here: R0 just off 0) and the
double-float ones."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sms():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


@pytest.fixture(scope="module")
def off_zero(torus64):
    return dataclasses.replace(torus64.geom, R0=1e-12), torus64.prims


def _size(rays):
    """The largest image of height 128 with at most this many rays, and one more column."""
    return (rays // 128, 128), (rays // 128 + 1, 128)


@pytest.mark.parametrize("prec,opts", [(0, {}), (0, {"no_sample_pool": 1}), (1, {})], ids=["pool", "in_place", "mixed"])
def test_renders_at_both_sides_of_the_line(off_zero, prec, opts):
    from raptor_gb300 import engine
    inside, outside = _size(5 * 128 * _sms())
    eng, ref = engine.Engine(**opts), engine.Engine(blocks_per_sm=2, **opts)
    ga, gb = eng.upload_grid(*off_zero), ref.upload_grid(*off_zero)
    for (w, h), one in ((inside, True), (outside, False)):
        kw = dict(stepsize=0.1, integrator=2)
        a, _ = eng.render(engine.image_desc(w, h, [230e9], grid=ga, **kw), prec)
        assert (eng.stats()["blocks_per_sm"] == 1) == one
        b, _ = ref.render(engine.image_desc(w, h, [230e9], grid=gb, **kw), prec)
        assert ref.stats()["blocks_per_sm"] == 2
        assert np.array_equal(a, b) and np.any(a)
    eng.close()
    ref.close()


@pytest.mark.parametrize("prec,opts,rays_per_lane", [(0, {}, 5), (0, {"no_sample_pool": 1}, 5), (1, {}, 2.5)],
                         ids=["pool", "in_place", "mixed"])
def test_adjoints_at_both_sides_of_the_line(off_zero, prec, opts, rays_per_lane):
    """A launch just beyond the line and its halves, both within it: the
    gradients are the halves' sums to the order of the sums (1e-12 in FP64;
    1e-5, some hundred roundings, in the FP32 transfer's)."""
    from raptor_gb300 import engine
    eng = engine.Engine(**opts)
    (w, h), (w1, _) = _size(int(rays_per_lane * 128 * _sms()))
    kw = dict(grid=eng.upload_grid(*off_zero), stepsize=0.1, integrator=2)
    tight = engine.image_desc(w, h, [230e9], **kw)
    eng.vjp(tight, np.ones(w * h), prec, want_fields=False)
    assert eng.stats()["grid_blocks"] == _sms()
    desc, n = engine.image_desc(w1, h, [230e9], **kw), w1 * h
    _, g = eng.vjp(desc, np.ones(n), prec, want_fields=False)
    assert eng.stats()["grid_blocks"] > _sms()
    _, lo = eng.vjp(desc, np.ones(n), prec, want_fields=False, ray_begin=0, ray_count=n // 2)
    assert eng.stats()["grid_blocks"] == _sms()
    _, hi = eng.vjp(desc, np.ones(n), prec, want_fields=False, ray_begin=n // 2, ray_count=n)
    eng.close()
    for key in ("d_m_unit", "d_r_high", "d_r_low", "d_inclination"):
        parts = abs(lo[key]) + abs(hi[key])
        assert abs(lo[key] + hi[key] - g[key]) <= (1e-12 if prec == 0 else 1e-5) * parts, key


@pytest.mark.parametrize("integrator,rays_per_lane", [(4, 2), (2, 1)], ids=["rk4", "rk2"])
def test_double_float_lines(torus64, integrator, rays_per_lane):
    from raptor_gb300 import engine
    inside, outside = _size(rays_per_lane * 128 * _sms())
    eng, ref = engine.Engine(), engine.Engine(blocks_per_sm=2)
    ga, gb = (e.upload_grid(torus64.geom, torus64.prims) for e in (eng, ref))
    for (w, h), one in ((inside, True), (outside, False)):
        kw = dict(stepsize=0.1, integrator=integrator)
        a, _ = eng.render(engine.image_desc(w, h, [230e9], grid=ga, **kw), engine.PREC_MIXED_DF)
        assert (eng.stats()["blocks_per_sm"] == 1) == one
        b, _ = ref.render(engine.image_desc(w, h, [230e9], grid=gb, **kw), engine.PREC_MIXED_DF)
        assert np.array_equal(a, b) and np.any(a)
    eng.close()
    ref.close()


@pytest.mark.parametrize("prec", [0, 1, 2], ids=["fp64", "mixed", "mixed_df"])
def test_a_range_takes_its_own_launch_rules(torus64, prec):
    """A small range of a large image is launched as a small image is, with the
    bits of the whole: every register budget of a form's kernel gives the same
    (FP64: 4, 3 and 2 blocks per SM, the others 3 and 2)."""
    from raptor_gb300 import engine
    eng = engine.Engine()
    w, h = 1024, 4 * _sms()
    desc = engine.image_desc(w, h, [230e9], grid=eng.upload_grid(torus64.geom, torus64.prims), stepsize=0.1)
    full, _ = eng.render(desc, prec)
    assert eng.stats()["blocks_per_sm"] > 1
    for rays_per_sm, one in ((100, True), (400, False), (1000, False), (2000, False)):
        count = rays_per_sm * _sms()
        begin = (w * h - count) // 2
        part, _ = eng.render(desc, prec, ray_begin=begin, ray_count=count)
        assert (eng.stats()["blocks_per_sm"] == 1) == one and eng.stats()["rays"] == count
        assert np.array_equal(part[begin:begin + count], full[begin:begin + count]) and np.any(part)
    eng.close()
