"""Which launch a call takes, by name, and the launch counter (scenarios in kernel_names.py)."""
import json
import os
import subprocess
import sys

import pytest

import kernel_names as K

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def seen():
    script = os.path.join(os.path.dirname(os.path.abspath(__file__)), "kernel_names.py")
    run = subprocess.run([sys.executable, script], capture_output=True, text=True, timeout=600)
    assert run.returncode == 0, run.stderr[-4000:]
    return json.loads(run.stdout.splitlines()[-1])


def _get(seen, key):
    if seen[key] is None:
        pytest.skip("the profiler has not seen all launches")
    return seen[key]


@pytest.mark.parametrize("case", list(K.SWEEPS), ids=str)
def test_line_solve(seen, case):
    n = _get(seen, "sweep %d %d %d %d %d" % case)
    sweeps = {k for k in n if k.startswith("sweep_")} - {"sweep_exact_kernel<double, true>", "sweep_exact_kernel<float, true>"}
    assert sweeps == {K.SWEEPS[case]}, n


@pytest.mark.parametrize("case", K.TUNING, ids=str)
def test_every_stride_times_the_pipelined_launch(seen, case):
    """The stride is the pipelined launch's, also on a domain small enough for the launch with
    every line in a warp, which has none."""
    prec, nx = case[:2]
    r = _get(seen, "tuning %d %d %d %d" % case)
    pipe = f"sweep_rb_pipe_kernel<{'double' if prec == 0 else 'float'}>"
    assert r["create"].get(pipe) == 12, r  # three strides, four rounds
    assert not any(k.startswith("sweep_resident_kernel") for k in r["create"]), r
    assert r["stride"] in (8, 16, 32)
    # and the solve itself is the one the domain calls for
    if r["step"] is not None:
        assert any(k.startswith("sweep_resident_kernel") for k in r["step"]) == (nx == 40), r
        assert (pipe in r["step"]) == (nx != 40), r


@pytest.mark.parametrize("case", K.SCHEMES, ids=str)
def test_assembly_form(seen, case):
    """The exponential scheme's A(0) is 0 / 0: it has no short form of a cell without flow, and
    the launch shapes made for that form are not for it."""
    scheme, prec, nx = case[:3]
    n = _get(seen, "scheme %s %d %d %d %d" % case)
    forms = [k.replace(" ", "") for k in n if k.startswith("energy_assemble_kernel")]
    t, dc = ("float" if prec == 1 else "double"), ("true" if prec == 2 else "false")
    if scheme == "exponential_law":
        want = f"{t},2,{dc},false,{3 if prec == 1 else 2}"
    else:
        want = f"{t},1,{dc},{'false' if nx == 60 else 'true'},{2 if prec != 1 else 4 if nx == 200 else 3}"
    assert forms == [f"energy_assemble_kernel<{want}>"], n


@pytest.mark.parametrize("case", K.COUNTS, ids=str)
def test_launch_counter(seen, case):
    for counted, launches in _get(seen, "count %d %d %d %s" % case):
        assert counted == launches


def test_powder_bed_grows_out_of_the_resident_launch(seen):
    """250x60 cells in FP64: 64 planes of 30 slots fit 148 CTAs of 13 (224 KB of rows), the 68
    planes with the second layer do not."""
    forms = [{k.split("<")[0] for k in n if k.startswith("sweep_")} for n in _get(seen, "powder")]
    assert forms == [{"sweep_resident_kernel"}] * 3 + [{"sweep_rb_pipe_kernel"}] * 2, forms
