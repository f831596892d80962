"""What the library's host code enqueues, and in which order, on a runtime without a GPU."""
import pytest

import host_runtime


@pytest.fixture(scope="module")
def library(tmp_path_factory):
    return host_runtime.build(tmp_path_factory.mktemp("host"))


START = """
import numpy as np
def solver(n, scale=1, fft="fp32"):
    s = pkg.Solver.create(n=n, dyeScale=scale, fft=fft)
    s.configure({"beta": 0.0, "drag": 0.0, "viscosity": 1.0, "hyperP": 2, "forceAmp": 0.0, "forceK": 20.0,
                 "forceWidth": 2.0, "cfl": 0.5, "dtMin": 1e-6, "dtMax": 1e-3, "dyeFade": 1.0})
    s.reset({"k0": 6, "amplitude": 3, "seed": 5, "dyePattern": "none"})
    return s
def kernels(rec):
    return [op[2][0] for op in rec.ops if op[0] == "kernel"]
"""


def test_a_pack_is_unblocked_once(library):
    """4096^2, packs of an earlier phase, no room on the device and the second pack's transfer fails:
    the first pack, already in rows, is not rewritten by the read that follows, and the next step
    makes the packs again."""
    host_runtime.run(library, START + """
s = solver(4096)
s.step(1, dye=False)
s.phase = 0
def read(name):
    try:
        s.getBuffer(name)
        return True
    except pkg.S2DError:
        return False
pkg.host.host_fail(b"cudaMallocAsync", 0, 2)
pkg.host.host_fail(b"upload", 1, 1)
pkg.host.host_forget()
assert not read("packA")
ups = [op[2][0] for op in Record(pkg.host).ops if op[0] == "upload"]
assert len(ups) == 1
pkg.host.host_fail(b"cudaMallocAsync", 0, 2)
pkg.host.host_forget()
assert read("packA")
again = [op[2][0] for op in Record(pkg.host).ops if op[0] == "upload"]
assert len(again) == 1 and again != ups, (ups, again)
pkg.host.host_forget()
s.encodeStep()
names = kernels(Record(pkg.host))
assert sum("k_pair_rows" in k for k in names) == 4, names    # three stages, and the packs before them
s.encodeStep()
assert sum("k_pair_rows" in k for k in kernels(Record(pkg.host))) == 7
""")


@pytest.mark.parametrize("call", ["s.getBuffer('packA')", "s.nlPack()", "s.fft.forward(None, 'packB')", "s.velocityPack(0)",
                                  "s.seedPhysical(np.ones(4096 * 4096, np.float32))"])
def test_calls_on_the_packs_allocate_nothing(library, call):
    """4096^2, the packs of the current state: put in rows without device memory for a second copy and
    without a way through host memory."""
    host_runtime.run(library, START + f"""
s = solver(4096)
s.step(1, dye=False)
pkg.host.host_fail(b"cudaMallocAsync", 0, 1)
pkg.host.host_forget()
{call}
rec = Record(pkg.host)
moved = [op for op in rec.ops if op[0] in ("upload", "copy") and int(op[2][2]) > 1 << 26]
assert not moved, moved
s.encodeStep()
""")


@pytest.mark.parametrize("n,scale,fft", [(256, 1, "tc-f16"), (256, 2, "tc-bf16"), (512, 2, "tc-f16"), (1024, 1, "tc-f16"),
                                         (64, 2, "fp32"), (256, 2, "fp32"), (512, 2, "fp32"), (1024, 2, "fp32")])
def test_the_dye_branch_joins_before_the_next_velocity(library, n, scale, fft):
    """Graphs of six substeps: every dye kernel is ordered behind the kernel that writes its velocity
    and ahead of the next one that does, whichever kernels a solver steps with."""
    host_runtime.run(library, START + f"""
s = solver({n}, {scale}, {fft!r})
s.step(1)
pkg.host.host_forget()
s.step(6, graph=True)
rec = Record(pkg.host)
dye = rec.find("kernel", "k_dye_fused")
one, columns = rec.find("kernel", "k_pair_step"), rec.find("kernel", "cols")
writers = rec.find("kernel", "k_nl_pack") or one or columns[2::3]
assert len(dye) == 6 and len(writers) in (6, 18), (dye, writers)
for d in dye:
    for w in writers:
        assert rec.ordered(d, w), (d, w, rec.ops[d], rec.ops[w])
last = rec.find("graph")[-1]
assert max(dye) < last
""")


@pytest.mark.parametrize("calls", ["s.encodeStep(); s.encodeReduce()", "s.encodeReduce()", "s.step(1, dye=False)",
                                   "s.step(1, dye=False, graph=True)"])
def test_the_copied_time_step_is_not_one_that_a_later_step_writes(library, calls):
    """copyDiagnostics, then steps and reductions that write both dt slots: whatever reads a slot on
    another stream is ordered ahead of them."""
    host_runtime.run(library, START + f"""
pkg.host.host_forget()
s = solver(64)
slots = [int(op[2][0]) for op in Record(pkg.host).ops if op[0] == "set" and int(op[2][1]) == 16]
assert len(slots) == 1
s.step(2, dye=False)
pkg.host.host_forget()
s.encodeDiagnostics(); s.copyDiagnostics()
for _ in range(3):
    {calls}
rec = Record(pkg.host)
copies = rec.find("download")
assert copies
reads = [i for i in copies if int(rec.ops[i][2][1]) < slots[0] + 16 and int(rec.ops[i][2][1]) + int(rec.ops[i][2][2]) > slots[0]]
writers = [i for i in rec.find("kernel") + rec.find("graph") if i > copies[-1]]
assert writers
for r in reads:
    for w in writers:
        assert rec.ordered(r, w), (rec.ops[r], rec.ops[w])
""")


@pytest.mark.parametrize("after", [0, 1, 2])
def test_a_read_goes_on_where_a_helper_thread_cannot_start(library, after):
    """A field read by several threads, memory short as the second, third or fourth is made: their
    shares fall to the threads that run, and no exception leaves the call."""
    host_runtime.run(library, START + f"""
s = solver(2048)
want = np.arange(2048 * 2048, dtype=np.float32).astype(np.complex64).reshape(2048, 2048)
want[683:1366], want[:, 683:1366] = 0, 0
s.setBuffer("state0", want)
assert np.array_equal(s.getBuffer("state0"), want)      # the slots are made
pkg.host.host_fail_new({after})
got = s.getBuffer("state0")
pkg.host.host_fail_new(-1)
assert np.array_equal(got, want)
""")


def test_a_solver_without_readback_slots_reads_directly(library):
    """Memory short as the slots' holder is made (the second allocation of create): the solver works,
    and so does one made and destroyed beside it."""
    host_runtime.run(library, START + """
pkg.host.host_fail_new(1)
s = pkg.Solver.create(n=64, dyeScale=1)
pkg.host.host_fail_new(-1)
t = solver(2048)
w = np.zeros((64, 64), np.complex64); w[1, 1] = 3
s.setBuffer("state0", w)
for _ in range(3):
    assert np.array_equal(s.getBuffer("state0"), w) and t.getBuffer("state0").shape == (2048, 2048)
s.destroy()
assert t.getBuffer("state0").shape == (2048, 2048)
t.destroy()
""")


def test_short_runs_do_not_capture_at_every_place(library):
    """Runs of seven substeps start at every place of the cycle of six: the first captures a graph of
    six, the others go on with single ones, until these have cost what a capture does."""
    host_runtime.run(library, START + """
def calls(s, runs):
    pkg.host.host_forget()
    for n in runs:
        s.step(n, graph=True)
    lines = pkg.host.host_record().decode().splitlines()
    return sum(l.startswith("captured") for l in lines), sum(l.startswith("graph") for l in lines)
for scale in (1, 2):
    s = solver(64, scale)
    assert calls(s, [7]) == (2, 2)                   # six, one
    assert calls(s, [7] * 5)[0] == 5                 # the single substeps of the other places
    calls(s, [7] * 300)
    assert calls(s, [7] * 6) == (0, 12)              # in the end a six and a single one each
s = solver(256)
assert calls(s, [100]) == (5, 20)                    # 16 sixes, four single ones, captured where they lie
assert calls(s, [100]) == (2, 20)                    # two single ones to the graph, 16 sixes, two more
""")
