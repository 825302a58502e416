"""The bench's clock sampler goes on under load after a timed region that is shorter
than its sampling period, until a line has come or its limit is over."""
import time

import pytest

import bench


class Running:  # stands for the nvidia-smi process
    def poll(self):
        return None


LINE = "GPU-aaa, 1965, 1965, 650.0, 0x0, Not Active, Not Active, Not Active, Not Active\n"


@pytest.fixture
def sampler(monkeypatch):
    monkeypatch.setattr(bench, "torch_sync", lambda: None)
    s = bench.ClockSampler("GPU-aaa")
    s.proc, s.skip = Running(), 1
    s.path.write_text(LINE)  # the priming line
    return s


def test_steps_until_a_line_comes(sampler):
    steps = []

    def step():
        steps.append(1)
        if len(steps) == 3:
            with open(sampler.path, "a") as f:
                f.write(LINE)

    sampler.settle(step)
    assert len(steps) == 3
    c = sampler.summary()
    assert c["samples"] == 1 and c["sm_mhz"] == 1965.0 and c["reasons"] == []


def test_no_step_where_the_region_was_sampled(sampler):
    sampler.path.write_text(2 * LINE)
    sampler.settle(lambda: pytest.fail("a line had come"))
    assert sampler.summary()["samples"] == 1


def test_gives_up(sampler):
    t0 = time.perf_counter()
    sampler.settle(lambda: time.sleep(0.01), max_seconds=0.1)
    assert 0.1 <= time.perf_counter() - t0 < 1.0
    assert sampler.summary()["reasons"] == ["no samples"]
