"""A sweep runs its steps and nothing else by default: the trial steps of
Batch.autotune choose nothing, take a copy of the whole state and force a list
rebuild, so they come only where they are asked for."""
import numpy as np
import pytest

from spsslangevinintegration_gb300 import surrogate, sweep

POINTS = [dict(n=64, sigma=1.0, D=0.1, m=1.0, density=2.0, R=1.0, v0=0.5)] * 3


class Recorder:
    def __init__(self, systems):
        self.systems = systems
        self.calls = []

    def autotune(self, *args, **kw):
        self.calls.append("autotune")

    def run(self, *args, **kw):
        self.calls.append("run")

    def stats(self):
        return np.zeros((self.systems, 5))

    def close(self):
        self.calls.append("close")


@pytest.fixture
def made(monkeypatch):
    batches = []

    def make(points, **kw):
        batches.append(Recorder(len(points)))
        return batches[-1]

    monkeypatch.setattr(sweep, "make_batch", make)
    return batches


def test_sweep_and_simulate_run_only_their_steps(made):
    sweep.run_sweep(POINTS, steps=20)
    surrogate.simulate(POINTS, steps=20, max_systems=2)
    assert [b.calls for b in made] == [["run", "close"]] * 3


def test_trial_steps_where_they_are_asked_for(made):
    sweep.run_sweep(POINTS, steps=20, autotune=True)
    surrogate.simulate(POINTS, steps=20, autotune=True)
    assert [b.calls for b in made] == [["autotune", "run", "close"]] * 2
