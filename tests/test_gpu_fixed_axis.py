"""Views along the polar axis at the top of the fixed-point geodesic's hslope
range, where its axis terms are largest, against the oracle port and, for the
mixed forms, the FP64 render."""
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


@pytest.mark.parametrize("hslope,inclination,integrator", [(1.8, 3.0, 4), (1.8, 175.0, 4), (1.6, 4.0, 2)])
def test_axis_views_match_port(eng, hslope, inclination, integrator):
    """48x41 rays over 40 M: at hslope 1.8 one in 50 passes the axis where a
    term of k^2 needs the widest format.  The mixed adjoint takes the same
    steps: its gradients meet the FP64 adjoint's at test_gpu_vjp.py's 2e-3."""
    from oracle import port
    from raptor_gb300 import engine, synth
    d = synth.make_torus(n1=64, n2=64, hslope=hslope)
    kw = dict(inclination=inclination, integrator=integrator)
    desc = engine.image_desc(48, 41, [230e9], grid=eng.upload_grid(d.geom, d.prims), **kw)
    img, spec = eng.render(desc, engine.PREC_FP64)
    ref = port.Scene(d.geom, d.prims, 48, 41, **kw).render([230e9])[0][:, 0]
    assert_fp64_parity(img, ref, f"hslope {hslope} at {inclination}")
    mixed, mspec = eng.render(desc, engine.PREC_MIXED)
    assert abs(mspec[0] - spec[0]) <= FLUX_RTOL_MIXED * abs(spec[0])
    bright = ref > 1e-2 * np.max(ref)
    assert np.max(np.abs(mixed[bright] / ref[bright] - 1.0)) <= 1e-2
    w = img / np.sum(img * img)
    _, g = eng.vjp(desc, w, engine.PREC_FP64)
    _, m = eng.vjp(desc, w, engine.PREC_MIXED)
    for key in ("d_m_unit", "d_r_high", "d_r_low", "d_inclination"):
        scale = max(abs(g[key]), 1e-6 * abs(g["d_r_high"]))
        assert abs(m[key] - g[key]) <= 2e-3 * scale, (key, m[key], g[key])


# hslope 0.3: the render's line at a camera x2 of 2^-13 lies at 0.037 degrees
@pytest.mark.parametrize("inclination", [0.03, 0.05, 179.95, 179.97])
def test_both_sides_of_the_renders_line(eng, torus64, inclination):
    from oracle import port
    from raptor_gb300 import engine
    desc = engine.image_desc(24, 21, [230e9], grid=eng.upload_grid(torus64.geom, torus64.prims),
                             inclination=inclination)
    img, spec = eng.render(desc, engine.PREC_FP64)
    ref = port.Scene(torus64.geom, torus64.prims, 24, 21, inclination=inclination).render([230e9])[0][:, 0]
    assert_fp64_parity(img, ref, f"{inclination} degrees")
    mixed, mspec = eng.render(desc, engine.PREC_MIXED)
    assert abs(mspec[0] - spec[0]) <= FLUX_RTOL_MIXED * abs(spec[0])


# and the mixed adjoint's, of 2^-8, at 1.2 degrees
@pytest.mark.parametrize("tape", [0, -1], ids=["one_pass", "two_passes"])
@pytest.mark.parametrize("inclination", [1.1, 1.3, 178.7, 178.9])
def test_both_sides_of_the_adjoints_line(torus64, inclination, tape):
    from raptor_gb300 import engine
    e = engine.Engine(vjp_tape=tape)
    desc = engine.image_desc(32, 31, [230e9], grid=e.upload_grid(torus64.geom, torus64.prims),
                             inclination=inclination, m_unit=1e19)
    img, _ = e.render(desc, engine.PREC_FP64)
    w = img / np.sum(img * img)
    _, g = e.vjp(desc, w, engine.PREC_FP64)
    out, m = e.vjp(desc, w, engine.PREC_MIXED)
    e.close()
    assert np.max(np.abs(out - img)) <= 1e-3 * np.max(img)
    for key in ("d_m_unit", "d_r_high", "d_r_low", "d_inclination"):
        scale = max(abs(g[key]), 1e-6 * abs(g["d_r_high"]))
        assert abs(m[key] - g[key]) <= 2e-3 * scale, (key, m[key], g[key])


def test_mixed_inclination_gradient_over_views(eng):
    """d_inclination of the mixed adjoint, FP32 tangents beside the fixed-point
    path, over twelve views of three grids: within 1e-5 of the FP64 adjoint's in
    the median (its FP32 sample alone leaves 4e-6, three hundred steps' FP32
    roundings some 1e-6), where a cancelling sum may leave single views further
    off."""
    from raptor_gb300 import engine, synth
    rng = np.random.default_rng(12)
    errors = []
    for k in range(12):
        d = synth.make_torus(n1=64, n2=64, hslope=(0.3, 1.0, 1.8)[k % 3])
        gid = eng.upload_grid(d.geom, d.prims)
        n = 40 + 2 * k
        desc = engine.image_desc(n, n + 1, [230e9], grid=gid, inclination=float(rng.uniform(10, 170)),
                                 integrator=4 if k % 4 else 2, m_unit=1e19)
        w = 1.0 + 0.3 * rng.standard_normal(n * (n + 1))
        g, m = (eng.vjp(desc, w, p, want_fields=False)[1]["d_inclination"] for p in (0, 1))
        errors.append(abs(m / g - 1.0))
    assert np.median(errors) <= 1e-5, errors


@pytest.mark.parametrize("size,inclination", [((33, 18), 20.0), ((33, 17), 90.0)])
def test_axis_column_without_spin(eng, size, inclination):
    """The middle column of an odd width looks along the axis.  Without spin its
    rays' k^phi is 0 and they end on the axis at the step cap; they are counted
    as in the FP64 geodesic (R0 of 1e-300, which changes no r), none non-finite."""
    import dataclasses
    from raptor_gb300 import engine, synth
    d = synth.make_torus(n1=64, n2=64, a=0.0)
    counts, images = [], []
    for geom in (d.geom, dataclasses.replace(d.geom, R0=1e-300)):
        desc = engine.image_desc(*size, [230e9], grid=eng.upload_grid(geom, d.prims), inclination=inclination)
        with pytest.warns(engine.EngineWarning):
            images.append(eng.render(desc, engine.PREC_FP64)[0])
        st = eng.stats()
        counts.append([st[k] for k in ("steps", "n_nonfinite", "n_stepcap")])
    assert counts[0] == counts[1] and counts[0][1] == 0 and counts[0][2] > 0, counts
    assert np.max(np.abs(images[0] - images[1])) <= 1e-9 * np.max(images[1])
