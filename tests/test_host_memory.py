"""What portions do with device memory, on the CPU: the library runs over tests/cudart_stub.cpp (no kernels; device memory is host
memory under a limit), each case in a process of its own."""
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

from cuqwen_b200 import binfmt, build
from cuqwen_b200 import stackfmt as F
import mixer_util
import stack_util

ROOT = Path(__file__).resolve().parent.parent
TABLE = dict(vocab=512, dim=256, inter=512, layers=2, heads=2, kv=1, hd=128, tied=True)
PRELUDE = """
import ctypes, os, sys
import numpy as np
from cuqwen_b200 import CuQwenError
from cuqwen_b200 import engine as E
stub = ctypes.CDLL(os.environ["LD_PRELOAD"])
stub.stub_limit.argtypes = [ctypes.c_size_t]
stub.stub_used.restype = stub.stub_peak.restype = ctypes.c_size_t
stub.stub_unordered.restype = ctypes.c_long
stub.stub_copies.restype = stub.stub_launches.restype = ctypes.c_char_p
copies = lambda: [int(n) for n in stub.stub_copies().split()]
toks = np.arange(20000, dtype=np.int32) % 50
"""


@pytest.fixture(scope="module")
def run(built, tmp_path_factory):
    """run(code, *args): a fresh interpreter with the stub in place of the CUDA runtime; its standard output."""
    lib = tmp_path_factory.mktemp("stub") / "libcudart_stub.so"
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", f"-I{build.cuda_home() / 'include'}", str(ROOT / "tests" / "cudart_stub.cpp"), "-o", str(lib)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr

    def go(code, *args):
        r = subprocess.run([sys.executable, "-c", PRELUDE + code, *map(str, args)], capture_output=True, text=True, timeout=300, cwd=ROOT,
                           env={**os.environ, "LD_PRELOAD": str(lib), "PYTHONPATH": str(ROOT)})
        assert r.returncode == 0, r.stdout + r.stderr
        return r.stdout
    return go


@pytest.fixture(scope="module")
def directories(tmp_path_factory):
    out = {}
    for name, cfg, w in (("falivik", stack_util.small(), None), ("gipotar", mixer_util.small(), mixer_util.weights("small", 11)[1])):
        out[name] = F.write_model_dir(tmp_path_factory.mktemp(name), cfg, w or stack_util.weights(cfg, 11)[0])
    return out


@pytest.fixture(scope="module")
def table_file(tmp_path_factory):
    path = tmp_path_factory.mktemp("table") / "m.bin"
    binfmt.write_model(path, TABLE, 2, binfmt.random_tensors(TABLE, 3))
    return path


@pytest.mark.parametrize("act", ["float32", "bfloat16"])
@pytest.mark.parametrize("design", ["falivik", "gipotar"])
def test_nothing_runs_beside_a_fill_of_its_workspace(run, directories, design, act):
    """The engine's stream does not wait for the default stream: a workspace that grows is cleared on the stream that uses it."""
    run("""
eng = E.Engine.open(sys.argv[1], act=sys.argv[2], max_seq_len=5200)
stub.stub_unordered()
at = 0
for n in (300, 700, 4100):
    eng.extend(toks[:n], at, [n - 1])
    assert stub.stub_unordered() == 0, n
    at += n
""", directories[design], act)


OPEN = {"table": """
def make(max_seq):
    eng = E.Engine(E.custom_params(512, 256, 512, 2, 2, 1, 128, 2, max_seq_len=max_seq))
    eng.load(sys.argv[1])
    return eng
longest = 8192
""", "directory": """
def make(max_seq):
    return E.Engine.open(sys.argv[1], act=sys.argv[2], max_seq_len=max_seq)
longest = 4096
"""}
ENGINES = [("table", ""), ("falivik", "bfloat16"), ("gipotar", "float32"), ("gipotar", "bfloat16")]


@pytest.fixture(scope="module")
def run_engine(run, directories, table_file):
    def go(name, act, code):
        path = table_file if name == "table" else directories[name]
        return run(OPEN["table" if name == "table" else "directory"] + code, path, act)
    return go


@pytest.mark.parametrize("name,act", ENGINES)
def test_a_prompt_is_cut_where_the_largest_workspace_does_not_fit(run_engine, name, act):
    run_engine(name, act, """
eng = make(9000)
eng.prefill(toks[:256], 0)
small = stub.stub_used()
eng.prefill(toks[:longest], 0)
large = stub.stub_used()
eng.close()
copies()
eng = make(9000)
eng.prefill(toks[:2], 0)                                       # 256 rows
base = stub.stub_used()
per_row = (large - small) / (longest - 256)
stub.stub_limit(base + int(1500 * per_row))                    # room for some 1500 rows more than those
copies()
eng.prefill(toks[:5000], 0)
cut = [n // 4 for n in copies()]
assert sum(cut) == 5000 and 1024 <= max(cut) <= 1800 and len(cut) <= 5, cut
eng.prefill(toks[:5000], 0)                                    # asked again: what stands does
assert [n // 4 for n in copies()] == cut
stub.stub_limit(1 << 40)
eng.prefill(toks[:5000], 0)
assert [n // 4 for n in copies()] == [min(5000, longest)] + [5000 - longest] * (longest < 5000)
""")


@pytest.mark.parametrize("name,act", ENGINES)
def test_a_workspace_that_stands_is_not_given_up_for_one_that_does_not_fit(run_engine, name, act):
    run_engine(name, act, """
eng = make(9000)
eng.prefill(toks[:2000], 0)
stub.stub_limit(stub.stub_used())                              # another program holds the rest
held = stub.stub_used()
copies(); stub.stub_peak()
for n in (2100, 4000, 9000):
    eng.prefill(toks[:n], 0)
    cut = [c // 4 for c in copies()]
    assert sum(cut) == n and cut[0] == 2048, cut
    assert stub.stub_used() == stub.stub_peak() == held
""")


@pytest.mark.parametrize("name,act", ENGINES)
def test_a_workspace_is_no_longer_than_the_cache(run_engine, name, act):
    run_engine(name, act, """
eng = make(3000)
eng.prefill(toks[:3000], 0)
all_of_it = stub.stub_used()
eng.close()
eng = make(3000)
for n in (300, 2100, 2400):
    eng.prefill(toks[:n], 0)
    assert stub.stub_used() <= all_of_it, n
""")


@pytest.mark.parametrize("name,act", ENGINES)
def test_no_room_at_all_is_an_error_and_the_next_call_starts_clean(run_engine, name, act):
    run_engine(name, act, """
eng = make(3000)
stub.stub_limit(stub.stub_used())
try:
    eng.prefill(toks[:700], 0)
    raise SystemExit("a portion without a workspace")
except CuQwenError as e:
    assert "memory" in str(e), e
stub.stub_limit(1 << 40)
copies()
eng.prefill(toks[:700], 0)
assert [c // 4 for c in copies()] == [700]
""")
