"""The engine's host code on a CUDA runtime without a device
(fake_cudart.cpp, preloaded into a child process): what its calls queue, record
and wait for, and what they leave behind when a runtime call fails."""
import functools
import os
import subprocess
import sys

import pytest

from awsemmd_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))

OFFSET = """
#include <cstdio>
#include "awsem_kernels.cuh"
int main() { printf("%d", (int) (sizeof(awsem::dev::NLState) - offsetof(awsem::dev::NLState, overflow))); }
"""

PRELUDE = """
import ctypes, sys, tempfile
sys.path.insert(0, {root!r})
from awsemmd_b200 import engine, synth
fake = ctypes.CDLL({lib!r})
for name in ("pending", "capturing", "graphs", "execs", "instantiated", "waits"):
    getattr(fake, "fake_" + name).restype = ctypes.c_longlong
ff = synth.forcefield_dir(tempfile.mkdtemp(dir={tmp!r}))
def chain(n, seed=1):
    return synth.chain_arrays(n, seed, n_mem_per_window=2)
def system(n=20, precision="fp64"):
    return engine.AwsemBatch.from_arrays(ff, [chain(n)], precision=precision)
def refused(call):
    try:
        call()
    except engine.AwsemError:
        return True
    return False
"""


@pytest.fixture(scope="module")
def host(gpu_lib, tmp_path_factory):
    d = tmp_path_factory.mktemp("host")
    lib = str(d / "fake_cudart.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-o", lib, os.path.join(HERE, "fake_cudart.cpp")], check=True)

    @functools.cache
    def overflow():
        (d / "o.cu").write_text(OFFSET)
        inc = ["-I" + os.path.join(os.path.dirname(HERE), p) for p in ("awsemmd_b200/csrc", "include")]
        subprocess.run([build.nvcc(), "-std=c++17", "--expt-relaxed-constexpr", *build.ARCH, *inc, "-o", str(d / "o"), str(d / "o.cu")],
                       check=True)
        return subprocess.run([str(d / "o")], check=True, capture_output=True, text=True).stdout

    def run(script):
        script = script.replace("OVERFLOW_FROM_END", overflow()) if "OVERFLOW_FROM_END" in script else script
        code = PRELUDE.format(root=os.path.dirname(HERE), lib=lib, tmp=str(d)) + script
        r = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, LD_PRELOAD=lib), capture_output=True, text=True,
                           timeout=300)
        assert r.returncode == 0, r.stdout + r.stderr

    return run


@pytest.mark.parametrize("what,call", [("compute", "cudaMemcpyAsync"), ("compute", "cudaEventRecord"),
                                       ("compute", "cudaLaunchKernel"), ("compute", "cudaGraphInstantiate"),
                                       ("run", "cudaEventRecord"), ("run", "cudaLaunchKernel"),
                                       ("run", "cudaGraphInstantiate")])
def test_failed_recording(what, call, host):
    """A runtime call that fails while a call's graph is recorded: the capture
    is over, no graph is left behind, a force call is evaluated without one,
    and the next call works."""
    host(f"""
what, call = {what!r}, {call!r}.encode()
s = system()
x = s.get_state(0)[0]
one = (lambda: s.compute(x)) if what == "compute" else (lambda: s.run(30))
for after in range({{b"cudaMemcpyAsync": 2, b"cudaGraphInstantiate": 1}}.get(call, 3)):
    s.set_launch_shapes((1, 148, 148, 0))  # drops what is recorded
    fake.fake_fail(call, after, 1)
    for k in range(100):
        no = refused(one)
        assert fake.fake_capturing() == 0 and fake.fake_graphs() == 0, (after, k)
        if fake.fake_failed(call):
            break
    assert fake.fake_failed(call), after
    assert no == (what == "run"), after
    assert not refused(one), after
""")


@pytest.mark.parametrize("what", ["compute", "run", "set_state", "get_state", "energies", "forces", "serve"])
def test_failed_call_is_over_when_it_returns(what, host):
    """A copy that fails in the middle of a call: nothing of the call is still
    queued on the handle's buffers when it returns, and the next call works."""
    host(f"""
what = {what!r}
if what == "serve":
    s = engine.AwsemServer(ff, 256, 4, 1 << 16)
    def one():
        slot = s.admit(chain(20), 3)
        s.advance(4)
        s.collect(slot)
else:
    s = system()
    x, v = s.get_state(0)
    s.compute(x)
    one = dict(compute=lambda: s.compute(x), run=lambda: s.run(2), set_state=lambda: s.set_state(x, v),
               get_state=lambda: s.get_state(0), energies=lambda: s.energies(0), forces=lambda: s.forces(0))[what]
hit = 0
for after in range(3 if what == "serve" else 8):
    fake.fake_fail(b"cudaMemcpyAsync", after, 0)
    no = refused(one)
    assert no == bool(fake.fake_failed(b"cudaMemcpyAsync")), after
    hit += no
    assert fake.fake_pending() == 0, after
    fake.fake_fail(b"cudaMemcpyAsync", 10 ** 6, 0)
    assert not refused(one), after
assert hit
""")


def test_collected_request_has_left_the_device(host):
    """The residues and memory tables of a collected request are cleared when
    the call returns: other entry points read them on other streams."""
    host("""
s = engine.AwsemServer(ff, 256, 4, 1 << 16)
slots = [s.admit(chain(20, k), 3) for k in range(3)]
s.advance(4)
for slot in slots:
    s.collect(slot)
    assert fake.fake_pending() == 0
""")


def test_request_is_collected_whole(host):
    """A collection waits once; one that fails before it has cleared the
    request leaves it to be collected again."""
    host("""
s = engine.AwsemServer(ff, 256, 4, 1 << 16)
for call in (b"", b"cudaMemcpyAsync", b"cudaLaunchKernel"):
    for after in range(4):
        slot = s.admit(chain(20, after), 3)
        s.advance(4)
        natoms = dict(s.natoms)
        if call:
            fake.fake_fail(call, after, 0)
        waits = fake.fake_waits()
        no = refused(lambda: s.collect(slot))
        if no:
            s.natoms = natoms
            assert s.usage()["requests"] == 1
            fake.fake_fail(call, 10 ** 6, 0)
            waits = fake.fake_waits()
            s.collect(slot)
        assert no == (bool(call) and after < {b"cudaMemcpyAsync": 4, b"cudaLaunchKernel": 2}[call]), (call, after)
        assert fake.fake_waits() == waits + 1 and fake.fake_pending() == 0
        assert s.usage()["requests"] == 0
""")


@pytest.mark.parametrize("pattern", [[7], [7, 1], [7, 7, 7, 1], [1, 1, 1, 2, 2, 2], [1, 2, 3, 4, 5, 6, 7]])
def test_force_calls_record_once(pattern, host):
    """A few force calls record nothing; many record one graph for each set of
    terms, in whatever turn a host asks for them, until the handle drops them."""
    host(f"""
pattern = {pattern!r}
s = system()
x = s.get_state(0)[0]
for t in set(pattern):
    for k in range(5):
        s.compute(x, terms=t)
assert fake.fake_instantiated() == 0
for k in range(60):
    for t in pattern:
        s.compute(x, terms=t)
assert fake.fake_instantiated() == fake.fake_execs() == len(set(pattern))
s.set_launch_shapes((1, 148, 148, 0))
assert fake.fake_execs() == 0
s.compute(x, terms=pattern[0])
assert fake.fake_execs() == 0
""")


def test_runs_record_what_they_use(host):
    """A first short run records single steps only, a long one those and the
    graph of 25; short windows again and again get the graph of five."""
    host("""
with system() as s:
    s.run(20)
    assert fake.fake_instantiated() == 1
    for k in range(10):
        s.run(19)
    assert fake.fake_instantiated() == 1
    for k in range(20):
        s.run(3, thermo=True)  # its graphs are made anew for every run
        s.run(19)
    assert fake.fake_instantiated() == 2 + 20
    s.run(30, thermo=True)
    assert fake.fake_instantiated() == 2 + 20 + 2
    for k in range(400):
        s.run(9, thermo=True)
    assert fake.fake_instantiated() == 2 + 20 + 2 + 400
    s.set_launch_shapes((1, 148, 148, 0))
    s.run(20)
    assert fake.fake_execs() == 1
""")


@pytest.mark.parametrize("after", range(4))
def test_pair_list_that_cannot_grow(after, host):
    """No memory for a larger pair list: the call that needed it fails, the
    handle keeps the list it had."""
    host(f"""
s = system()
x = s.get_state(0)[0]
s.compute(x)
capacity = s.model_info()[5]
assert capacity > 0
fake.fake_patch(OVERFLOW_FROM_END, 10 ** 6)  # the evaluation reports an overflow
fake.fake_fail(b"cudaMalloc", {after}, 0)
assert refused(lambda: s.compute(x))
assert fake.fake_failed(b"cudaMalloc")
assert s.model_info()[5] == capacity
assert not refused(lambda: s.compute(x))
fake.fake_patch(OVERFLOW_FROM_END, 10 ** 6)
s.compute(x)
assert s.model_info()[5] == 2 * 10 ** 6
""")
