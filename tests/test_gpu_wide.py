"""FP64 renders against the port in long double (oracle/wide.py): the image
whose geodesic runs in fixed point is as close to more than 64 bits as the one
whose geodesic runs in FP64, which the FP64 VJP returns from the same transfer
sample.

The two images share the sample's roundings (2e-12) and differ by their
paths': where the fixed-point path is no worse, the root mean square, the
median and the upper decile of the pixels' errors agree to the spread of such
figures over some 450 pixels, for which half as much again is allowed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# inclination, step parameter, integrator: ordinary views, views along the
# axis, where fixed point resolves the angle least, and small steps there
@pytest.mark.parametrize("inclination,stepsize,integrator", [(60.0, 0.05, 4), (17.0, 0.05, 2), (2.0, 0.05, 4),
                                                             (1.0, 0.05, 2), (1.0, 0.01, 4), (1.0, 0.01, 2),
                                                             (1.0, 0.003, 2)])
def test_fixed_point_is_as_close_as_fp64(torus64, inclination, stepsize, integrator):
    from oracle import wide
    from raptor_gb300 import engine
    w, h = 24, 21
    kw = dict(inclination=inclination, stepsize=stepsize, integrator=integrator)
    ref = wide.render(torus64.geom, torus64.prims, w, h, [230e9], **kw)[:, 0]
    bright = ref > 1e-6 * ref.max()
    eng = engine.Engine()
    desc = engine.image_desc(w, h, [230e9], grid=eng.upload_grid(torus64.geom, torus64.prims), **kw)
    image, _ = eng.render(desc, engine.PREC_FP64)
    stepped, _ = eng.vjp(desc, np.ones(w * h), engine.PREC_FP64, want_fields=False)
    eng.close()
    figures = []
    for im in (image, stepped):
        err = (im[bright] - ref[bright]).astype(np.float64)
        rel = np.abs(err / ref[bright].astype(np.float64))
        figures.append((np.sqrt(np.mean(err ** 2)), np.median(rel), np.quantile(rel, 0.9)))
    for fixed, fp64 in zip(*figures):
        assert fixed <= 1.5 * fp64, figures
