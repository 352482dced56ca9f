"""How the planner's probe times a launch, on a device whose clock the test keeps: an event into an idle
stream is recorded before the host has issued the launch that follows it, events are 2 us apart at the
finest, and now and then a launch takes longer."""
import numpy as np
import pytest

DEVICE_US = 41.0   # what a launch takes
ISSUE_US = 9.0     # what the host takes to issue one


class Device:
    def __init__(self):
        self.busy, self.n, self.rng = False, 0, np.random.default_rng(5)

    def launch(self):
        """One launch; its time between events as they come out."""
        self.n += 1
        us = DEVICE_US + self.rng.uniform(0, 2) + (8.0 if self.n % 10 == 0 else 0.0) + (900.0 if self.n % 37 == 0 else 0.0)
        us += 0.0 if self.busy else ISSUE_US
        self.busy = True
        return 2.0 * round(us / 2.0) / 1e3

    def sync(self):
        self.busy = False


@pytest.mark.parametrize("whole_block", [True, False])
def test_probe_times_the_device_alone(monkeypatch, whole_block):
    import es_learned
    import es_native as N
    dev = Device()

    class Ctx:
        capacity = 1 << 20
        n_outer = 1 << 12 if whole_block else 1 << 40

        @classmethod
        def from_arrays(cls, *a):
            return cls()

        def launch(self, *a):
            dev.launch()

        def launch_timed(self, *a):
            ms = dev.launch()
            dev.sync()
            return ms

        def stage_counts(self):
            dev.sync()
            return np.ones(2, dtype=np.uint64)

        set_block = set_tune = reset = reset_counts = close = lambda self, *a: None

    class Batch:
        def __init__(self, *a):
            pass

        def run(self, use_graph):
            self.ms = dev.launch()

        def sync(self):
            dev.sync()
            return self.ms

        def close(self):
            pass

    monkeypatch.setattr(N, "Context", Ctx)
    monkeypatch.setattr(N, "Batch", Batch)
    monkeypatch.setattr(N.PlanArrays, "from_arrays", classmethod(lambda cls, *a: None))
    arrays = (12, np.array([32]), None, None, np.array([7, 11]), None, 1)
    got = [es_learned.probe({"arrays": arrays}, {"layout": 5}, 20)["ms"] * 1e3 for _ in range(20)]
    assert max(got) < DEVICE_US + 4.0 and min(got) > DEVICE_US - 1.0
