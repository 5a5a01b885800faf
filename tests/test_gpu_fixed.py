"""The fixed-point geodesic on the GPU: renders at both sides of every line of
the rule that picks it, and of those that pick its launch.

A pixel may differ from the oracle port by the FP64 bar (parity.py); on these
small images that allows no grazing pixel, so the cameras see the torus from
outside the critical curve's finest orders (24x21 pixels over 40 M).  A batch
and its parts run the same arithmetic per ray, so the launch rules change no
bit within one kernel and at most last bits between two register budgets."""
import numpy as np
import pytest

from tests.parity import FLUX_RTOL_MIXED, assert_fp64_parity

pytestmark = pytest.mark.gpu


@pytest.fixture
def eng():
    from raptor_gb300 import engine
    e = engine.Engine()
    yield e
    e.close()


# fixed point covers 0.2 <= hslope <= 1.8 and steps of 1e-7 to 0.1
EDGES = [dict(hslope=0.2), dict(hslope=0.19), dict(hslope=1.0), dict(hslope=1.8), dict(hslope=1.81),
         dict(stepsize=0.1), dict(stepsize=0.101), dict(stepsize=0.02), dict(a=0.1), dict(a=0.5), 
         dict(a=0.998), dict(inclination=2.0), dict(inclination=177.0), dict(camera=1, inclination=75.0),
         dict(integrator=2), dict(integrator=2, inclination=5.0, stepsize=0.03)]


@pytest.mark.parametrize("edge", EDGES, ids=[",".join(f"{k}={v}" for k, v in e.items()) for e in EDGES])
def test_rule_edges_match_port(eng, edge):
    from oracle import port
    from raptor_gb300 import engine, synth
    d = synth.make_torus(n1=64, n2=64, **{k: v for k, v in edge.items() if k in ("a", "hslope")})
    kw = dict(inclination=50.0, **{k: v for k, v in edge.items() if k not in ("a", "hslope", "inclination")})
    kw["inclination"] = edge.get("inclination", 50.0)
    gid = eng.upload_grid(d.geom, d.prims)
    desc = engine.image_desc(24, 21, [230e9], grid=gid, **kw)
    img, spec = eng.render(desc, engine.PREC_FP64)
    ref, _, rs = port.Scene(d.geom, d.prims, 24, 21, **kw).render([230e9], with_stats=True)
    st = eng.stats()
    assert st["rays"] == 24 * 21 and st["n_nonfinite"] == 0
    assert abs(st["steps"] - int(rs["steps"].sum())) <= 0.001 * st["steps"]
    assert np.any(ref != 0)
    assert_fp64_parity(img, ref[:, 0], str(edge))
    if edge.get("a") == 0.1:
        return  # a flux of 1e-44 Jy, below the FP32 sample's range with either geodesic
    mixed, mspec = eng.render(desc, engine.PREC_MIXED)
    assert abs(mspec[0] - spec[0]) <= FLUX_RTOL_MIXED * abs(spec[0])


@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "mixed"])
def test_two_register_budgets_agree(eng, torus64, prec):
    """2^19 rays run the 4-block kernel, each half of them the 3-block one;
    both are compiled from one source and agree at the FP64 bar (the mixed
    form's FP32 sample to 1e-5 of the brightest pixel)."""
    from raptor_gb300 import engine
    gid = eng.upload_grid(torus64.geom, torus64.prims)
    descs = [engine.image_desc(512, 512, [230e9], grid=gid, inclination=i, stepsize=0.1) for i in (60.0, 110.0)]
    both, _ = eng.render(descs, prec)
    assert eng.stats()["rays"] == 1 << 19
    one = np.concatenate([eng.render(d, prec)[0] for d in descs])
    if prec == 0:
        assert_fp64_parity(both, one, "two budgets")
    else:
        assert np.max(np.abs(both - one)) <= 1e-5 * np.max(one)


@pytest.mark.parametrize("prec", [0, 1, 2], ids=["fp64", "mixed", "mixed_df"])
@pytest.mark.parametrize("w,h", [(330, 333), (331, 340), (608, 512)])
def test_queue_order_covers_every_ray(eng, torus64, prec, w, h):
    """Launches of 5/4 to 8 lanes' worth of rays hand rays out from the middle
    of the image: each ray once, its pixel as in a render of it alone in a
    small range (which keeps the plain order)."""
    from raptor_gb300 import engine
    gid = eng.upload_grid(torus64.geom, torus64.prims)
    d = engine.image_desc(w, h, [230e9], grid=gid, inclination=70.0, stepsize=0.1)
    full, _ = eng.render(d, prec)
    assert eng.stats()["rays"] == w * h
    n = w * h
    for begin, count in ((0, 33), (n // 2 - 50, 101), (n - 65, 65), (n // 3, 3000)):
        part, _ = eng.render(d, prec, ray_begin=begin, ray_count=count)
        assert np.array_equal(part[begin:begin + count], full[begin:begin + count])
    assert np.any(full[:n // 2]) and np.any(full[n // 2:])


@pytest.mark.parametrize("case", [dict(inclination=4.0), dict(inclination=176.0), dict(camera=1),
                                  dict(integrator=2, stepsize=0.1), dict(hslope=1.8), dict(hslope=1.81)],
                         ids=["pole", "south", "log", "rk2", "fixed_edge", "fp64_edge"])
def test_mixed_adjoint_matches_fp64(eng, case):
    """The mixed adjoint's geodesic and tangents in fixed point against the
    FP64 adjoint, at the 2e-3 that test_gpu_vjp.py holds it to."""
    from raptor_gb300 import engine, synth
    d = synth.make_torus(n1=64, n2=64, hslope=case.get("hslope", 0.3))
    gid = eng.upload_grid(d.geom, d.prims)
    kw = dict(grid=gid, inclination=55.0, m_unit=1e19)
    kw.update({k: v for k, v in case.items() if k != "hslope"})
    desc = engine.image_desc(32, 31, [230e9], **kw)
    img, _ = eng.render(desc, engine.PREC_FP64)
    w = img / np.sum(img * img)
    _, g = eng.vjp(desc, w, engine.PREC_FP64)
    _, m = eng.vjp(desc, w, engine.PREC_MIXED)
    for key in ("d_m_unit", "d_r_high", "d_r_low", "d_inclination"):
        scale = max(abs(g[key]), 1e-6 * abs(g["d_r_high"]))
        assert abs(m[key] - g[key]) <= 2e-3 * scale, (key, m[key], g[key])


@pytest.mark.parametrize("prec,inside,outside", [(0, (170, 171), (171, 171)), (1, (197, 197), (198, 197)),
                                                 (2, (197, 197), (198, 197))], ids=["fp64", "mixed", "mixed_df"])
def test_small_launches_take_one_block_per_sm(eng, torus64, prec, inside, outside):
    """At both sides of the line the launch's shape changes no bit."""
    from raptor_gb300 import engine
    ref = engine.Engine(blocks_per_sm=2)
    ga, gb = (e.upload_grid(torus64.geom, torus64.prims) for e in (eng, ref))
    lanes = 0
    for size, blocks in ((inside, 1), (outside, 2)):
        a, _ = eng.render(engine.image_desc(*size, [230e9], grid=ga, stepsize=0.1), prec)
        st = eng.stats()
        lanes = st["grid_blocks"] // st["blocks_per_sm"] * st["block_size"]
        if lanes == 152 * 128:
            assert st["blocks_per_sm"] == blocks
        b, _ = ref.render(engine.image_desc(*size, [230e9], grid=gb, stepsize=0.1), prec)
        assert np.array_equal(a, b) and np.any(a)
    ref.close()


def test_fp64_adjoint_grids_agree(eng, torus64):
    """312x312 rays are more than five per lane of one block per SM, its halves
    fewer: the image's gradients are the halves' sums, to the order of the
    FP64 sums (1e-12)."""
    from raptor_gb300 import engine
    gid = eng.upload_grid(torus64.geom, torus64.prims)
    desc = engine.image_desc(312, 312, [230e9], grid=gid, inclination=60.0, stepsize=0.1)
    w = np.ones(312 * 312)
    _, g = eng.vjp(desc, w, engine.PREC_FP64, want_fields=False)
    whole = eng.stats()["grid_blocks"]
    half = 312 * 156
    _, lo = eng.vjp(desc, w, engine.PREC_FP64, want_fields=False, ray_begin=0, ray_count=half)
    assert eng.stats()["grid_blocks"] * 2 == whole or whole != 2 * 152
    _, hi = eng.vjp(desc, w, engine.PREC_FP64, want_fields=False, ray_begin=half, ray_count=half)
    for key in ("d_m_unit", "d_r_high", "d_r_low", "d_inclination"):
        parts = abs(lo[key]) + abs(hi[key])
        assert abs(lo[key] + hi[key] - g[key]) <= 1e-12 * parts, key
