"""The trainer's error flag and its first state, in a child process (fake_cudart.c)
that sets the flag as a bounded wait would and delays what the host does not wait for."""
import pytest

from tests.fake_cudart import run_child

pytestmark = pytest.mark.gpu

HEAD = """
import numpy as np
import freeshearlayer_b200 as fsl
rng = np.random.default_rng(1)
X = rng.uniform(0.1, 1.0, (1000, 8)).astype(np.float32)
Y = rng.uniform(0.0, 0.1, 1000).astype(np.float32)

def trainer():
    t = fsl.Trainer(1024, seed=3)
    t.set_samples(X, Y)
    return t, fake.small()

def give_up(flag):
    one = ctypes.c_int(1)
    assert ctypes.CDLL("libcudart.so.12").cudaMemcpy(ctypes.c_void_p(flag), ctypes.byref(one), ctypes.c_size_t(4), 1) == 0

def timed_out(call):
    try:
        call()
    except fsl.FslError as e:
        return e.code == -5  # FSL_ERR_TIMEOUT
    return False
"""


def test_passes_after_the_flag_do_nothing():
    run_child(HEAD + """
t, flag = trainer()
w = t.weights()
for n in (1000, 128, 1):
    give_up(flag)
    assert timed_out(lambda: t.gradient(n))
give_up(flag)
assert timed_out(lambda: t.train(2, 256))
assert np.array_equal(t.weights(), w)
""")


@pytest.mark.parametrize("first", ["train", "gradient", "set_weights"])
def test_a_reported_flag_is_cleared_and_its_steps_not_counted(first):
    run_child(HEAD + f"""
t, flag = trainer()
t.train(2, 256)
give_up(flag)
if {first!r} == "set_weights":
    t.set_weights(t.weights())
else:
    assert timed_out(lambda: t.train(3, 256) if {first!r} == "train" else t.gradient())
u, _ = trainer()
u.train(2, 256)
if {first!r} == "set_weights":
    u.set_weights(u.weights())
a, b = t.gradient(), u.gradient()
assert a[1] == b[1] and np.array_equal(a[0], b[0])
assert t.train(2, 256) == u.train(2, 256)  # the same Adam step count, too
assert np.array_equal(t.weights(), u.weights())
""")


def test_a_new_trainer_waits_for_its_first_state():
    run_child(HEAD + """
u, _ = trainer()
fake.late(True)
t, _ = trainer()
a = t.train(2, 256)
fake.late(False)
assert a == u.train(2, 256) and np.array_equal(t.weights(), u.weights())
""")
