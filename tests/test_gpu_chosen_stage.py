"""Which FP64 stage kernel runs, counted in a child process (fake_cudart.c): the grid's
choice, the tuning calls that set it aside and bring it back, and the ensembles
that capture it."""
import pytest

from tests.fake_cudart import run_child

pytestmark = pytest.mark.gpu

HEAD = """
import time
import numpy as np
import freeshearlayer_b200 as fsl
from tests.helpers import random_state, spatial_params, temporal_params

DIR, RING = "k_stage_dir", "k_stageI"

def domain(L, H, D, setup="temporal", **kw):
    p = temporal_params(L, H, D, deltaT=1e-6, **kw) if setup == "temporal" else spatial_params(L, H, D)
    d = fsl.Domain(p)
    d.upload_state(random_state(p, 11))
    return d, p

def ran(call):
    fake.reset()
    call()
    return fake.count(DIR), fake.count(RING)
"""


# grids on either side of the rule (148 SMs); the ring in both setups, its last
# segment and its last tiles ragged
@pytest.mark.parametrize("L,H,D,setup,ring", [(64, 32, 32, "temporal", False), (37, 56, 30, "temporal", True),
                                              (77, 27, 57, "temporal", True), (40, 30, 30, "spatial", True)])
def test_the_grids_choice_equals_oracle(L, H, D, setup, ring):
    run_child(HEAD + f"""
from oracle import oracle as orc
orc.build()
d, p = domain({L}, {H}, {D}, {setup!r})
assert ran(lambda: d.step(2)) == ((0, 6) if {ring} else (6, 0))
o = orc.Oracle(p)
o.set_state(random_state(p, 11))
o.step(2)
assert np.all(np.isfinite(o.state())) and np.array_equal(d.download_state(), o.state())
""")


def test_ensemble_captures_again_after_tuning_a_member():
    run_child(HEAD + """
d, _ = domain(64, 32, 32)
e = fsl.Ensemble([d])
e.set_chunk(2)
e.step(5)
fake.reset()
e.step(4)
assert fake.graphs() == 0
d.tune(d.TUNE_STAGE_SEG, 32)  # the value it has by default
assert ran(lambda: e.step(4)) == (0, 6) and fake.graphs() == 1
e.sync()
""")


def test_ensemble_tuner_measures_the_grids_choice():
    run_child(HEAD + """
d, _ = domain(64, 32, 32)
d.tune(d.TUNE_STAGE_SEG, 20)
e = fsl.Ensemble([d])
fake.reset()
rows, seg, _ = e.tune(trial_steps=2)
assert fake.count(DIR) == 9  # one plain step and one captured chunk of two
assert ran(lambda: d.step(1)) == ((3, 0) if rows == 0 else (0, 3))
e.sync()
""")


def test_rows_zero_returns_to_the_grids_choice():
    run_child(HEAD + """
d, _ = domain(64, 32, 32)
assert ran(lambda: d.step(1)) == (3, 0)
d.tune(d.TUNE_STAGE_SEG, 16)
assert ran(lambda: d.step(1)) == (0, 3)
d.tune(d.TUNE_STAGE_ROWS, 0)
assert ran(lambda: d.step(1)) == (3, 0)
d.tune(d.TUNE_STAGE_ROWS, 0)
d.tune(d.TUNE_STAGE_SEG, 16)
assert ran(lambda: d.step(1)) == (0, 3)
""")


def test_a_long_domains_launches_cost_the_host_little():
    # 2^20 planes: a search over every segment length takes milliseconds, and a step
    # needs a dozen of its results
    run_child(HEAD + """
d, _ = domain(1 << 20, 2, 2, deltaX=1.0, deltaY=1.0, deltaZ=1.0)
d.step(1)
d.sync()
best = 1e9
for _ in range(3):
    t0 = time.perf_counter()
    d.step(1)
    best = min(best, time.perf_counter() - t0)
    d.sync()
assert best < 5e-3, best
""")
