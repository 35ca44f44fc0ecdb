"""Host logic of the entry points without a GPU, failed allocations among it: the library runs
in a child process whose CUDA runtime calls go to a host stand-in (fake_cudart.c) that
records kernel launches and fails the allocation it is told to."""
import json
import os
import subprocess
import sys
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    so = tmp_path_factory.mktemp("fake") / "libfakecudart.so"
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-o", str(so), str(HERE / "fake_cudart.c")], check=True)
    return so


PRELUDE = """
import ctypes as C, json, sys
sys.path[:0] = [{lib!r}, {oracle!r}, {tests!r}]
import numpy as np
from dmrgb200 import _capi as capi, engine as E, models as M, mps as S
fake = C.CDLL({so!r})
fake.fake_live.restype = C.c_long

def launched():
    out = []
    for i in range(fake.fake_launches()):
        k, g, b = C.c_ulong(), C.c_uint(), C.c_uint()
        fake.fake_launch(i, C.byref(k), C.byref(g), C.byref(b))
        out.append([k.value, g.value, b.value])
    fake.fake_clear()
    return out
"""


def child(fake, body):
    pre = PRELUDE.format(lib=str(HERE.parent / "maquis-dmrg_b200"), oracle=str(HERE.parent / "oracle"),
                         tests=str(HERE), so=str(fake))
    res = subprocess.run([sys.executable, "-c", pre + body], capture_output=True, text=True, timeout=300,
                         env={**os.environ, "LD_PRELOAD": str(fake)})
    assert res.returncode == 0, res.stdout + res.stderr
    return json.loads(res.stdout.strip().splitlines()[-1])


PLAN = """
from helpers import make_chain
from test_lowering import hpsi_plan
model, bonds, _, _ = make_chain("hubbard", 12, 0, seed=1, synthetic_m=60)
plan = hpsi_plan(model, bonds, 5)
assert E.lowering(plan).chained
n = max(int(plan["in_size"]), int(plan["out_size"]))
store = np.zeros(1 << 16)
nl, nr = int(plan["c_ci"].max()) + 1, int(plan["t_ci"].max()) + 1
addr = lambda k: np.full(k, store.ctypes.data, np.uint64)
x, y = np.zeros(n), np.zeros(n)
make = lambda: E.DevicePlan(E.Context(0), plan, left_addr=addr(nl), other_addr=addr(nr))
"""


def test_host_buffer_program_lowered_again_after_a_failed_allocation(fake):
    """Host-buffer H·psi of a chained plan whose GEMM variants are then pinned: whichever
    allocation of the new lowering fails, the call says so, and the next one launches what a
    fresh pinned plan launches (it must not run on a half-lowered program)."""
    got = child(fake, PLAN + """
p = make()
p.set_gemm_variants(0, 0)
fake.fake_clear()
p.hpsi_host(x.ctypes.data, y.ctypes.data)
want = launched()
rows = []
for k in range(1, 200):
    p = make()
    p.hpsi_host(x.ctypes.data, y.ctypes.data)
    chained = launched()
    p.set_gemm_variants(0, 0)
    fake.fake_fail_in(k)
    status = 0
    try:
        p.hpsi_host(x.ctypes.data, y.ctypes.data)
    except capi.DmrgError as e:
        status = e.status
    fake.fake_fail_in(0)
    first = launched()
    p.hpsi_host(x.ctypes.data, y.ctypes.data)
    rows.append([status, first == want, launched()])
    if status == 0:
        break
print(json.dumps({"want": want, "chained": chained, "rows": rows}))
""")
    want, rows = got["want"], got["rows"]
    assert len(got["chained"]) < len(want) and got["chained"] != want
    assert rows[-1][0] == 0 and len(rows) > 8
    for status, same, later in rows[:-1]:
        assert status == 3  # out of memory
        assert later == want


def test_host_buffer_first_call_after_a_failed_allocation(fake):
    """The same at the first host-buffer call (program, device vectors, streams, events, graph),
    and destroying the plan gives everything back."""
    got = child(fake, PLAN + """
p = make()
fake.fake_clear()
p.hpsi_host(x.ctypes.data, y.ctypes.data)
want = launched()
del p
rows = []
for k in range(1, 200):
    before = fake.fake_live()
    p = make()
    fake.fake_fail_in(k)
    status = 0
    try:
        p.hpsi_host(x.ctypes.data, y.ctypes.data)
    except capi.DmrgError as e:
        status = e.status
    fake.fake_fail_in(0)
    launched()
    p.hpsi_host(x.ctypes.data, y.ctypes.data)
    rows.append([status, launched()])
    del p
    rows[-1].append(fake.fake_live() - before)
    if status == 0:
        break
print(json.dumps({"want": want, "rows": rows}))
""")
    want, rows = got["want"], got["rows"]
    assert rows[-1][0] == 0 and len(rows) > 8
    for status, later, leaked in rows[:-1]:
        assert status == 3 and later == want and leaked == 0


def test_autotuning_ends_a_pin(fake):
    """Pinned variants replace a plan's chained products by its stages; autotuning the plan
    brings the one launch back, from device and from host buffers."""
    got = child(fake, PLAN + """
p = make()
a = x.ctypes.data, y.ctypes.data
dev = lambda: (fake.fake_clear(), p.hpsi(*a), launched())[-1]
host = lambda: (fake.fake_clear(), p.hpsi_host(*a), launched())[-1]
out = [dev(), host()]
p.set_gemm_variants(0, 0)
out += [dev(), host()]
capi.check(capi.lib.dmrgb200_plan_autotune(p.handle, *a, None, None), "autotune")
out += [dev(), host()]
print(json.dumps(out))
""")
    dev, host, pinned, pinned_host, again, again_host = got
    assert len(dev) == 1 and len(pinned) > 1 and pinned_host != host
    assert again == dev and again_host == host


STEP = """
from helpers import make_chain
from test_lowering import step_plan
model, bonds, _, _ = make_chain("hubbard", 12, 0, seed=1, synthetic_m={m})
plan = step_plan(model, bonds, 4, True)
assert bool(E.lowering(plan).chained) == {chained}
store = np.zeros(1 << 20)
nt, nc = int(plan["t_ci"].max()) + 1, int(plan["c_out_ci"].max()) + 1
far = np.full(nc, store.ctypes.data + (1 << 22), np.uint64) + 64 * np.arange(nc, dtype=np.uint64)
ket = np.zeros(int(plan["in_size"]))
bra = np.zeros(int(plan["out_size"]))
make = lambda: E.DevicePlan(E.Context(0), plan, left_addr=np.full(nt, store.ctypes.data, np.uint64))
run = lambda p, out=far: p.step(ket.ctypes.data, bra.ctypes.data, out)
"""


@pytest.mark.parametrize("m,chained", [(60, True), (700, False)])
def test_step_after_a_failed_allocation(fake, m, chained):
    """Whichever allocation of a step fails, the next call runs it as a fresh plan does, and
    destroying the plan gives everything back."""
    got = child(fake, STEP.format(m=m, chained=chained) + """
p = make()
fake.fake_clear()
run(p)
want = launched()
del p
rows = []
for k in range(1, 60):
    before = fake.fake_live()
    p = make()
    fake.fake_fail_in(k)
    status = 0
    try:
        run(p)
    except capi.DmrgError as e:
        status = e.status
    fake.fake_fail_in(0)
    launched()
    run(p)
    rows.append([status, launched()])
    del p
    rows[-1].append(fake.fake_live() - before)
    if status == 0:
        break
print(json.dumps([want, rows]))
""")
    want, rows = got
    assert (len(want) == 1) == chained
    assert rows[-1][0] == 0 and len(rows) >= (2 if chained else 4)
    for status, later, leaked in rows[:-1]:
        assert status == 3 and later == want and leaked == 0


def test_chained_step_over_its_input_runs_the_stages(fake):
    """A chained step whose output overlaps its ket or its boundary runs the stages, with
    their scratch allocated then; the next call elsewhere is one launch again."""
    got = child(fake, STEP.format(m=60, chained=True) + """
p = make()
out = []
for addr in (far, np.full(nc, ket.ctypes.data, np.uint64), far, np.full(nc, store.ctypes.data, np.uint64), far):
    a = fake.fake_allocations()
    fake.fake_clear()
    run(p, addr)
    out.append([len(launched()), fake.fake_allocations() - a])
print(json.dumps(out))
""")
    (n0, a0), (n1, a1), (n2, _), (n3, a3), (n4, _) = got
    assert n0 == n2 == n4 == 1 and n1 >= 3 and n3 >= 3
    assert a1 == a3 == a0 + 2  # T and S
