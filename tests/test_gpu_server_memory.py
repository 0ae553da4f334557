"""The server's admission estimate covers what a RIS job's frames allocate for ray queues, result
slots and light-candidate weights, over scenes whose BSDF rays matter too; a job is refused only
for what it cannot render without."""
import numpy as np
import pytest

from hdrestir_b200 import abi, configs
from hdrestir_b200.scene import Light
from hdrestir_b200.server import Server

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("reservoir", [True, False])
@pytest.mark.parametrize("dome", [True, False])
def test_admission_covers_the_weights(dome, reservoir):
    sc, cam = configs.config1(640, 480, n_lights=8)
    if dome:
        sc.lights.append(Light(abi.LIGHT_DOME, texture=np.full((4, 8, 3), 0.5, np.float32)))
    candidates, n_nee, n_bsdf = 32, 16, 16
    ris = dict(candidate_count=candidates, use_reservoir=reservoir, max_depth=1)
    frame = 96 + 16 + 16 + 16 + 49 + (80 if reservoir else 0)
    queues = n_nee * (32 + 1 + (4 if reservoir else 8)) + ((1 + n_bsdf) * (32 + 16 + 4) if dome else 0)
    charge = n_nee * 33 + (1 + n_bsdf) * 52
    with Server(device=0) as sv:
        sid = sv.add_scene(sc)
        sv.submit(sid, cam, 2, "ris", **ris)
        sv.submit(sid, cam, 2, "ris", **ris)
        sv.step()
        in_use = sv.load()[2]
    assert in_use >= 2 * 640 * 480 * (frame + queues)
    need = 640 * 480 * (frame + charge) + (1 << 20)
    with Server(device=0, hbm_budget=need) as sv:
        job = sv.submit(sv.add_scene(sc), cam, 1, "ris", **ris)
        assert sv.step() == 1
        assert np.isfinite(sv.take(job)).all()
    with Server(device=0, hbm_budget=need - 1) as sv:
        with pytest.raises(abi.HdrError):
            sv.submit(sv.add_scene(sc), cam, 1, "ris", **ris)
