"""GPU: networks that go through windows of steps by default, stepped one by one by the target-resident kernel all the same: what other
tests of that path say of them holds with the option "use_windows" at 0, too."""
import pytest

from genn_b200 import runtime
from tests import test_failure_paths, test_resident

pytestmark = pytest.mark.gpu

WINDOWED = ["ff_sparse", "ff_sparse_narrow", "ff_bitmask", "ff_dense", "cond_delay", "c1_full"]


@pytest.fixture(autouse=True)
def step_by_step(monkeypatch):
    """Every runtime that goes through windows is told not to; there has to be one in a test."""
    made = []

    class StepByStep(runtime.Runtime):
        def __init__(self, *args, **kwargs):
            super().__init__(*args, **kwargs)
            if self.counter("window_steps"):
                made.append(self)
            self.set_option("use_windows", 0)
            assert self.counter("window_steps") == 0

    monkeypatch.setattr(runtime, "Runtime", StepByStep)
    yield
    assert made


@pytest.mark.parametrize("ctas,warps", [(0, 0), (1, 24), (7, 4), (148, 24)])
@pytest.mark.parametrize("name", WINDOWED)
def test_all_steps_in_one_launch_match_the_reference(name, ctas, warps):
    test_resident.test_all_steps_in_one_launch_match_the_reference(name, ctas, warps)


@pytest.mark.parametrize("name", ["ff_sparse", "ff_bitmask", "cond_delay"])
def test_launches_of_every_length_hand_over_to_the_other_paths(name):
    test_resident.test_launches_of_every_length_hand_over_to_the_other_paths(name)


@pytest.mark.parametrize("synchronous", [False, True], ids=["patience 0", "more than the list holds"])
def test_a_busy_network_is_handed_over_and_taken_back(synchronous):
    test_resident.test_a_busy_network_is_handed_over_and_taken_back("late", synchronous)


def test_a_missing_message_runs_into_the_wait_limit():
    test_failure_paths.test_a_missing_message_of_the_target_resident_kernel_runs_into_the_wait_limit()
