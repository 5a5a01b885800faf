"""The FP64 VJP of a field close to the photon ring, whose rays circle the hole
and amplify a rounding of their path by some 500 per orbit: its adjoint steps
in FP64 where the render's geodesic is fixed point, so the image of the one
pass and the render agree to 1e-8 of the peak there.  In two passes the
adjoint reads each pixel's I from that render; its gradients stay within
test_gpu_vjp_tape.py's 1e-9 of the one pass's, in optically thin and thick
models."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m_unit", [1e19, 1e21])
@pytest.mark.parametrize("inclination", [17.0, 60.0])
def test_paths_of_circling_rays(torus64, inclination, m_unit):
    from raptor_gb300 import engine
    out = []
    for opts in ({}, {"vjp_tape": -1}, {"no_sample_pool": 1}):
        eng = engine.Engine(**opts)
        desc = engine.image_desc(96, 95, [86e9, 230e9], grid=eng.upload_grid(torus64.geom, torus64.prims), m_unit=m_unit,
                                 inclination=inclination, cam_size_x=11.0, cam_size_y=11.0)
        fwd, _ = eng.render(desc, engine.PREC_FP64)
        peak = float(np.max(fwd))
        image, g = eng.vjp(desc, (fwd / peak - 0.5) / fwd.size, engine.PREC_FP64)
        eng.close()
        assert float(np.max(np.abs(image - fwd))) <= 1e-8 * peak
        out.append(g)
    for g in out[1:]:
        for key in ("d_rho", "d_u", "d_lnthetae"):
            scale = float(np.max(np.abs(out[0][key])))
            assert scale > 0 and float(np.max(np.abs(g[key] - out[0][key]))) <= 1e-9 * scale, key
        for key in ("d_m_unit", "d_r_high", "d_r_low", "d_inclination"):
            assert g[key] == pytest.approx(out[0][key], rel=1e-9), key
