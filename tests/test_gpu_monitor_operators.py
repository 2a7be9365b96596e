"""The monitor between steps of the operator path reads the density that the step
stored: nothing is rebuilt, and the values are those of the rebuilt state."""
import pytest

from multiphaselb_b200 import abi
from tests.helpers import small_cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["cylinder_d2q9", "bubble_d2q9", "bubble_d3q15"])
def test_monitor_between_steps(gpu_lib, name):
    from multiphaselb_b200 import Lattice
    case = small_cases()[name]
    seen = []
    for rebuild in (False, True):
        with Lattice(case, path=abi.PATH_OPERATORS) as lat:
            lat.upload_case()
            lat.initialize()
            lat.monitor(reset=True)
            lat.step(1)
            got = [lat.monitor()]
            before = lat.info()["kernel_launches"]
            for n in (1, 2, 3):
                lat.step(n)
                if rebuild:
                    lat.download()
                got.append(lat.monitor())
            if not rebuild:  # two kernels a step, two a check
                assert lat.info()["kernel_launches"] - before == 2 * 6 + 2 * 3
            seen.append((got, lat.download()))
    assert seen[0][0] == seen[1][0]
    for k, v in seen[0][1].items():
        assert (v == seen[1][1][k]).all(), k
