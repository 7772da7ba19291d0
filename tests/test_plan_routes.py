"""A pricing plan chooses its kernel by the pairs of each run, not by the count it was made for (a rank prices its share
of a plan's pairs, a quote refines on the plan of an indication), and long schedules keep the specialised kernel: on the stand-in for the CUDA runtime, without a GPU."""

import pytest
from test_upload_order import on_the_stand_in  # noqa: F401 (the fixture)


# 148 SMs: rows beyond the stage are read with a pair's legs on two lanes (1000 pairs), streamed (16103 to 56831), or
# through L1; a table in the stage has no rows to stream
@pytest.mark.parametrize("n_x,routes", [(801, 3), (60, 2)], ids=["rows", "staged"])
@pytest.mark.parametrize("ladder", [False, True], ids=["autocall", "ladder"])
def test_a_runs_kernel_depends_on_its_own_pairs(on_the_stand_in, n_x, routes, ladder):  # noqa: F811
    on_the_stand_in(f"""
from optlab_b200._abi import OB_MODEL_PATHS
from optlab_b200.requests import mc_request
steps, n_x, ladder = 40, {n_x}, {ladder}
product = dict(product=0, leg_type=[1], leg_strike=[100.0], leg_barrier=[0], leg_level=[0.0], discount=1.0) if ladder \\
    else dict(product=1, obs_step=[steps], obs_discount=[1.0], trigger=[0.0], ki_barrier=0.6, put_strike=1.0)
fake.fake_first_kernel.restype = C.c_void_p

def plan(n_pairs):
    held = mc_request(model=OB_MODEL_PATHS, dt=np.full(steps, 1 / 252), t0=np.arange(steps) / 252, spot=[100.0],
                      n_pairs=n_pairs, seed=1, kind=[1], cvar=[0.0], root=np.eye(1), log_fwd=np.zeros((1, steps + 1)),
                      step_row=np.arange(steps)[None, :], lo=np.full(steps, -0.8), inv_dx=np.full(steps, (n_x - 1) / 1.6),
                      table=np.full((steps, n_x), 0.04), n_x=n_x, **product)
    p = C.c_void_p()
    check(lib.ob_mc_plan_create(C.byref(held.struct), 0, C.byref(p)))
    return p

def route(p, n_pairs):
    fake.fake_forget()
    check(lib.ob_mc_run(p, C.c_longlong(n_pairs), C.c_longlong(0), C.c_ulonglong(1), None))
    return fake.fake_first_kernel(), fake.fake_first_block()

counts = [1000, 16102, 16103, 30001, 56831, 56832, 2**19]
own = [route(plan(c), c) for c in counts]
assert len(set(k for k, _ in own)) == {routes}, own
for made_for in counts:
    p = plan(made_for)
    assert [route(p, c) for c in counts] == own, made_for
""")


@pytest.mark.parametrize("ladder", [False, True], ids=["autocall", "ladder"])
def test_a_heston_qe_request_of_thousands_of_steps_keeps_its_kernel(on_the_stand_in, ladder):  # noqa: F811
    # (27 years of daily steps: a double record of 32 bytes a step beside the step's tables passed the 220 KB stage)
    on_the_stand_in(f"""
from optlab_b200._abi import OB_MODEL_HESTON_QE
from optlab_b200.requests import mc_request
ladder = {ladder}
fake.fake_first_kernel.restype = C.c_void_p

def kernel(steps, precision):
    product = dict(product=0, leg_type=[1], leg_strike=[100.0], leg_barrier=[0], leg_level=[0.0], discount=1.0) if ladder \\
        else dict(product=1, obs_step=[steps], obs_discount=[1.0], trigger=[0.0], ki_barrier=0.6, put_strike=1.0)
    held = mc_request(model=OB_MODEL_HESTON_QE, dt=np.full(steps, 1 / 252), t0=np.arange(steps) / 252, spot=[100.0],
                      n_pairs=64, seed=1, heston=(0.04, 1.5, 0.04, 0.5, -0.7), r=0.02, q=0.0, **product)
    p = C.c_void_p()
    check(lib.ob_mc_plan_create(C.byref(held.struct), precision, C.byref(p)))
    fake.fake_forget()
    check(lib.ob_mc_run(p, C.c_longlong(64), C.c_longlong(0), C.c_ulonglong(1), None))
    return fake.fake_first_kernel()

for precision in (0, 1):
    assert len(set(kernel(steps, precision) for steps in (252, 6300, 6500, 6804))) == 1
""")
