"""Runs of test_gpu_launch_arms.py, as a program of their own: one named case,
its results written to a file."""
import os
import sys

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)

from fibrenet_b200 import generate as g  # noqa: E402
from fibrenet_b200.native import Simulation  # noqa: E402

FIELDS = ("pos", "img", "vel", "force", "vel_old")


def tensile(fibres, pull=0.5, cell=2.5):
    side = 1000.0 * np.sqrt(fibres / 20000.0)
    return g.tensile_network(seed=7, fibres=fibres, beads=50, box=(side, side, 20.0), clamp_lo=2.0,
                             clamp_hi=side - 2.0, pull=pull, cell=cell)


def state(s):
    count, partners = s.lists()
    return {**{f: s.get(f) for f in FIELDS}, "count": count, "partners": partners,
            **{f"status{k}": v for k, v in enumerate(s.status())}}


def steps(model, net=0, **kw):
    with Simulation(model, **kw) as s:
        for n in (1, 9, 16, 3):
            s.step(n)
        series = s.step_series(12, 5, energy=True, net=net)
        return {**state(s), "series": np.asarray(series), "rebuilds": s.stats()["rebuilds"]}


def gradients(model, **kw):
    with Simulation(model, **kw) as s:
        reaction = s.adjoint_forward(4, 10, 20, 1)
        grad = s.adjoint_backward(np.random.default_rng(3).normal(size=reaction.shape))
        return {**state(s), **grad, "reaction": reaction}


# a wave of blocks of the chain step holds about 73,000 beads; the incidence
# kernel's about as many
CASES = {
    "chain": lambda: steps(tensile(6100), list_capacity=32),
    "chain_small": lambda: steps(g.plain_network(seed=1, fibres=200, beads=50), list_capacity=32),
    "batch": lambda: steps([g.plain_network(seed=k, fibres=300 + 7 * k, beads=41, box=(120.0, 120.0, 10.0))
                            for k in range(12)], net=5, list_capacity=32),
    "incidence": lambda: steps(tensile(4000), chain=False, list_capacity=32),
    "displacement": lambda: steps(tensile(2500, pull=20.0, cell=3.0), verlet_skin=0.4, list_capacity=48),
    "gradients_chain": lambda: gradients(tensile(3000), list_capacity=32),
    "gradients_incidence": lambda: gradients(tensile(1500), chain=False, list_capacity=32),
}

if __name__ == "__main__":
    np.savez(sys.argv[2], **CASES[sys.argv[1]]())
