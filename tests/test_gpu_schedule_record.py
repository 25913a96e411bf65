"""engine_schedule_info() after job sets whose Krylov cycles run in one launch each."""
import pytest

import picuda
from tests import models as M

pytestmark = pytest.mark.gpu


def run(models):
    compiled = [picuda.compile(m) for m in models]
    rhos = [picuda.computational_product_state(m.basis, 2) for m in models]
    picuda.solve_dynamics_batch(compiled, rhos, (0.0, 0.1), saveat=0.05,
                                algorithm=picuda.ExpvAlgorithm(krylovdim=20, precision="mixed"))
    return picuda.engine_schedule_info()


def test_record_of_one_launch_cycles(lib_built):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    try:
        small = [M.scan_model(20, 0.9, 0.3, 0.1), M.scan_model(31, 0.9, 0.3, 0.1)]
        picuda.set_engine_schedule("per_tile")
        before = run(small)
        assert before["schedule"] == "per_tile" and before["items"] > 0
        picuda.set_engine_schedule("auto")
        info = run(small)
        assert info["schedule"] == "one_launch" and info["choices"] > before["choices"]
        assert info["items"] > 0 and info["resident_max"] >= 1
        assert info["candidates_us"] == {} and info["tunings"] == before["tunings"]
        large = run([M.scan_model(150, 0.9, 0.3, 0.1)])  # past the bound of one-launch sets
        assert large["schedule"] != "one_launch" and large["choices"] > info["choices"]
    finally:
        picuda.set_engine_schedule("auto")
