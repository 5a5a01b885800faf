"""The autotuner keeps a shape for launches of one kernel and one grid rule:
sizes on both sides of a line on the number of rays are tuned each for itself,
though their size class (a power of two) is the same."""
import pytest

pytestmark = pytest.mark.gpu


# the lines per SM: FP64 kernels of 2 and 3 blocks at 647 rays, mixed-DF ones at
# 1293; one block per SM up to 192 rays in FP64 and 256 in the others; the
# middle-out order up to 8 rays per lane (3 mixed blocks: 3072)
@pytest.mark.parametrize("prec,rays_per_sm", [(0, (470, 790)), (2, (920, 1580)), (0, (132, 210)), (1, (230, 395)),
                                              (2, (230, 395)), (1, (1725, 3200))],
                         ids=["fp64_budget", "df_budget", "fp64_grid", "mixed_grid", "df_grid", "mixed_order"])
def test_both_sides_of_a_line_are_tuned(torus64, tmp_path, monkeypatch, prec, rays_per_sm):
    import torch
    from raptor_gb300 import engine
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    cache = tmp_path / "tuned"
    monkeypatch.setenv("RAPTOR_TUNE_CACHE", str(cache))
    eng = engine.Engine(autotune=1)
    gid = eng.upload_grid(torus64.geom, torus64.prims)
    for rays in rays_per_sm:
        eng.render(engine.image_desc(rays * sms // 64, 64, [230e9], grid=gid, stepsize=0.1), prec)
    eng.close()
    keys = [line.split()[0] for line in cache.read_text().splitlines()]
    assert len(set(keys)) == len(keys) == 2, keys
