"""Every upload is ordered before the kernels that read it, whatever stream they run on, and the pinned staging keeps
working when it cannot grow: the engine library on a stand-in for the CUDA runtime (fake_cudart.cpp), without a GPU."""

import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent

HEAD = """
import ctypes as C, sys
import numpy as np
sys.path.insert(0, {package!r})
fake = C.CDLL({fake!r}, mode=C.RTLD_GLOBAL)
fake.fake_unordered.restype = C.c_char_p
fake.fake_host_limit.argtypes = [C.c_size_t]
fake.fake_pinned_bytes.restype = C.c_size_t
from optlab_b200 import engine, workloads
from optlab_b200._abi import check, load
from optlab_b200.requests import paths_request
lib = load()

def ordered(launches=1):
    assert fake.fake_launches() >= launches, fake.fake_launches()
    assert fake.fake_unordered() == b"", fake.fake_unordered().decode()
    fake.fake_forget()

def leverage(steps=6, n_lv=33):
    from optlab_b200.leverage import leverage_request
    h = leverage_request(dt=np.full(steps, 1 / 52), t0=np.arange(steps) / 52, n_pairs=512, seed=3,
                         heston=(0.04, 1.5, 0.04, 0.5, -0.7), n_x=21, lv_lo=np.full(steps, -1.0),
                         lv_inv_dx=np.full(steps, (n_lv - 1) / 2.0), lv_rows=np.full((steps, n_lv), 0.04), atm_vol=0.2)
    check(lib.ob_leverage(C.byref(h.struct), 0))

def columns(kinds=(1,), n_pairs=301, steps=5, n_x=11, n_obs=None, mixed=None):
    n, n_obs = len(kinds), steps if n_obs is None else n_obs
    h = paths_request(dt=np.full(steps, 1 / 52), t0=np.arange(steps) / 52, obs_step=np.arange(1, n_obs + 1),
                      root=np.eye(n), kind=list(kinds), cvar=np.full(n, 0.04),
                      heston=np.tile([0.04, 1.5, 0.04, 0.5, -0.7], n), same=1, fwd=np.full((n, n_obs), 100.0),
                      n_pairs=n_pairs, seed=5, step_row=np.tile(np.arange(steps), n), lo=np.full(steps, -0.5),
                      inv_dx=np.full(steps, n_x - 1.0), table=np.full((steps, n_x), 0.04), n_x=n_x)
    engine.paths(h, "fp32")
"""


@pytest.fixture(scope="module")
def on_the_stand_in(tmp_path_factory):
    """Runs code in a process of its own on the stand-in."""
    fake = tmp_path_factory.mktemp("fake") / "fake_cudart.so"
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", str(ROOT / "tests" / "fake_cudart.cpp"), "-o",
                    str(fake)], check=True)
    head = HEAD.format(package=str(ROOT / "option-pricing-lab_b200"), fake=str(fake))

    def run(code):
        r = subprocess.run([sys.executable, "-c", head + code], capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr[-2000:]

    return run


def test_the_stand_in_sees_a_launch_beside_an_upload_and_one_behind_it(on_the_stand_in):
    on_the_stand_in("""
a, s = C.c_void_p(), C.c_void_p()
fake.cudaStreamCreateWithFlags(C.byref(a), 1), fake.cudaStreamCreateWithFlags(C.byref(s), 1)
buf = (C.c_char * 64)()
for st, unordered in ((a, True), (s, False)):
    fake.cudaMemcpyAsync(buf, buf, C.c_size_t(64), 1, st)
    fake.cudaLaunchKernel(None, C.c_longlong(0), 0, C.c_longlong(0), 0, None, C.c_size_t(0), s)
    assert (fake.fake_unordered() != b"") == unordered
    fake.cudaStreamSynchronize(st)
    fake.fake_forget()
""")


def test_a_calibrations_inputs_are_ordered_before_its_kernels(on_the_stand_in):
    on_the_stand_in("leverage()\nordered()\nleverage()\nordered()\n")


@pytest.mark.parametrize("kinds,n_x", [((1,), 11), ((1,), 4001), ((0, 1), 11)], ids=["staged", "table", "generic"])
def test_path_columns_inputs_are_ordered_before_the_kernels_of_both_streams(on_the_stand_in, kinds, n_x):
    # (names of different kinds take the generic kernel; a column of 2^21 pairs goes in several chunks)
    on_the_stand_in(f"columns({kinds}, n_x={n_x})\nordered()\ncolumns({kinds}, n_x={n_x}, n_pairs=2**21, n_obs=1)\nordered(4)\n")


# (a plan is run on any stream its caller likes)
@pytest.mark.parametrize("n_x", [17, 801, 60001], ids=["staged", "small table", "large table"])
@pytest.mark.parametrize("generic", [False, True])
def test_a_plans_inputs_have_arrived_when_it_is_made(on_the_stand_in, generic, n_x):
    on_the_stand_in(f"""
import os
os.environ["OPTLAB_B200_GENERIC"] = "{int(generic)}"
w = workloads.worst_of(n_paths=512, years=0.25, steps_per_year=12, n_names=1, c=[0.03], rho=[-0.7], n_exp=3, n_x={n_x})
for precision in (0, 1):
    plan = C.c_void_p()
    check(lib.ob_mc_plan_create(C.byref(w.held.struct), precision, C.byref(plan)))
    assert fake.fake_outstanding() == 0
    check(lib.ob_mc_plan_destroy(plan))
""")


def test_an_adjoint_plans_inputs_have_arrived_when_it_is_made(on_the_stand_in):
    on_the_stand_in("""
from optlab_b200._abi import ObAdjointRequest
w = workloads.worst_of(n_paths=512, years=0.25, steps_per_year=12, n_names=1, c=[0.03], rho=[-0.7], n_exp=3, n_x=17)
rq = ObAdjointRequest()
rq.base, rq.smoothing = w.held.struct, 0.005
for precision in (0, 1):
    plan = C.c_void_p()
    check(lib.ob_adjoint_plan_create(C.byref(rq), precision, C.byref(plan)))
    assert fake.fake_outstanding() == 0
    check(lib.ob_adjoint_plan_destroy(plan))
""")


def test_a_books_inputs_have_arrived_when_it_is_made(on_the_stand_in):
    on_the_stand_in("""
from optlab_b200.batch import Batch, sample_book
Batch(sample_book(n_trades=4, seed=1, paths_log2=(8, 9), years=(1, 2)), "fp32")
assert fake.fake_outstanding() == 0
""")


SMALL, LARGE = 2 * 4 * 2**20, 2 * 32 * 2**20  # bytes of the two pairs of pinned slots


def test_a_pair_of_slots_that_cannot_grow_keeps_serving(on_the_stand_in):
    # a 1.3 MB table goes through the small pair; the columns of 2^23 pairs ask for the large one
    on_the_stand_in(f"""
table = dict(steps=40, n_x=4001, n_obs=1)
fake.fake_host_limit({SMALL})
columns(**table)
assert fake.fake_pinned_bytes() == {SMALL}
columns(n_pairs=2**23, n_obs=1)
columns(**table)
assert fake.fake_pinned_bytes() == {SMALL}
fake.fake_host_limit({LARGE})
check(lib.ob_release_buffers())
columns(**table)
columns(n_pairs=2**23, n_obs=1)
assert fake.fake_pinned_bytes() == {LARGE}
""")


def test_small_requests_after_a_refused_large_one_get_their_slots(on_the_stand_in):
    on_the_stand_in(f"""
fake.fake_host_limit({SMALL})
columns(n_pairs=2**23, n_obs=1)
assert fake.fake_pinned_bytes() == 0
columns(steps=40, n_x=4001, n_obs=1)
assert fake.fake_pinned_bytes() == {SMALL}
""")
