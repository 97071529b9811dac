"""A launch that the runtime refuses is reported by the call that makes it, for the
dynamic procedure and each stage of a step.  The refusal comes from a stand-in for the
runtime's launch calls (fake_cudart.c) in a child process; the device sees nothing of it."""
import pytest

from tests.fake_cudart import run_child

pytestmark = pytest.mark.gpu

HEAD = """
import numpy as np
import freeshearlayer_b200 as fsl
from tests.helpers import random_state, temporal_params

def refused(kernel, call, skip=0):
    fake.arm(kernel, skip)
    try:
        call()
    except fsl.FslError as e:
        assert e.code == -3, e  # FSL_ERR_CUDA
    else:
        raise AssertionError(kernel + " not launched and not reported")
    assert fake.refused() >= 1
    fake.arm("", 0)

def domain(**kw):
    p = temporal_params(24, 16, 20, deltaT=1e-6, **kw)
    d = fsl.Domain(p)
    d.upload_state(random_state(p, 3))
    return d

def weights(d):
    t = fsl.Trainer(1 << 14, seed=1)
    d.closure_set_scales(1e-3, 1.0)
    d.closure_set_weights(t.weights())
    return t
"""

DYNAMIC = {
    "phase": "d = domain(precision={prec}); refused('k_dyn_march', lambda: (d.ghost_bc(), d.dynamic_smagorinsky()))",
    "step": "d = domain(precision={prec}); refused('k_dyn_march', lambda: d.step(2))",
    "step, second": "d = domain(precision={prec}); refused('k_dyn_march', lambda: d.step(2), 1)",
    "phased": "d = domain(precision=0); refused('k_dyn_march', lambda: d.step_phased(1))",
    "stage": "d = domain(precision={prec}); refused('k_dyn_march', d.step_stage)",
    "judgement": "d = domain(precision={prec}, sgs=1); t = weights(d); d.closure_judge(1, 0.1); "
                 "refused('k_dyn_march', lambda: d.step(1))",
    "fallback": "d = domain(precision={prec}, sgs=1); t = weights(d); d.closure_judge(1000, 0.0); d.step(1); "
                "refused('k_dyn_march', lambda: d.step(1))",
    "compare": "d = domain(precision={prec}, sgs=1); t = weights(d); refused('k_dyn_march', d.closure_compare)",
    "harvest": "d = domain(precision={prec}); t = weights(d); refused('k_dyn_march', lambda: t.harvest(d))",
    "ensemble": "d = domain(precision={prec}); e = fsl.Ensemble([d]); e.step(1); e.set_chunk(2); "
                "refused('k_dyn_march', lambda: e.step(2))",
}


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("call", DYNAMIC)
def test_dynamic_procedure(call, prec):
    run_child(HEAD + DYNAMIC[call].format(prec=prec))

# the kernels a stage can take: FP64 direction split and ring, FP32 full lane and ring
@pytest.mark.parametrize("kernel,tune,prec", [("k_stage_dir", 0, 0), ("k_stageI", 16, 0), ("k_wide", 0, 1), ("k_stageI", 12, 1)])
@pytest.mark.parametrize("stage", [1, 2, 3])
def test_stages(kernel, tune, prec, stage):
    run_child(HEAD + f"""
d = domain(precision={prec})
d.tune(d.TUNE_STAGE_ROWS, {tune})
for s in (1, 2, 3):
    if s == {stage}:
        refused({kernel!r}, d.step_stage)
        break
    d.step_stage()
d = domain(precision={prec})
d.tune(d.TUNE_STAGE_ROWS, {tune})
refused({kernel!r}, lambda: d.step(1), {stage - 1})
""")
