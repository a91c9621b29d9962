"""Which engines run a step's layers as one kernel, and which launch by launch, on the CPU over tests/cudart_stub.cpp."""
import re
import subprocess
from pathlib import Path

import pytest

from cuqwen_b200 import binfmt, build
from test_host_memory import run                                           # noqa: F401  (fixture)

PLAIN = dict(vocab=512, dim=256, inter=512, layers=2, heads=4, kv=2, hd=64, tied=True)


def kernels_of_a_step(run, tmp_path, cfg, quant, flags="0", splits=0, sms=148):      # noqa: F811
    path = tmp_path / "m.bin"
    binfmt.write_model(path, cfg, quant, binfmt.random_tensors(cfg, 3))
    return run(f"""
stub.stub_sms({sms})
p = E.custom_params({cfg['vocab']}, {cfg['dim']}, {cfg['inter']}, {cfg['layers']}, {cfg['heads']}, {cfg['kv']}, {cfg['hd']}, {quant}, max_seq_len=256)
p.flags = E.FLAG_NO_GRAPH | {flags}
p.attn_splits = {splits}
eng = E.Engine(p)
eng.load(sys.argv[1])
stub.stub_launches()
eng.step(1, 0)
print(stub.stub_launches().decode())
assert eng.step_launches == (5 if "{flags}" == "0" and {splits} * {cfg['kv']} <= {sms} and {cfg['heads']} <= {sms} else 1 + 6 * {cfg['layers']} + 3)
""", path)


@pytest.mark.parametrize("quant", [0, 1, 2])
@pytest.mark.parametrize("hd", [64, 128])
def test_the_layers_of_a_step_are_one_launch(run, tmp_path, quant, hd):     # noqa: F811
    out = kernels_of_a_step(run, tmp_path, dict(PLAIN, hd=hd), quant).split("\n")
    names = [n for n in out if n]
    assert len(names) == 5 and "step_layers_kernel" in names[1] and " 148,1,1 " in names[1] and "gemv_kernel" in names[2]


@pytest.mark.parametrize("flags,splits,sms", [("E.FLAG_ACCURATE_ROPE", 0, 148), ("E.FLAG_SEPARATE_KERNELS", 0, 148), ("E.FLAG_NO_HANDOVER", 0, 148), ("E.FLAG_STEP_TRACE", 0, 148), ("E.FLAG_KV_INT8", 0, 148),
                                              ("0", 75, 148), ("0", 0, 3)])
def test_what_the_kernel_does_not_know_stays_launch_by_launch(run, tmp_path, flags, splits, sms):      # noqa: F811
    assert "step_layers_kernel" not in kernels_of_a_step(run, tmp_path, PLAIN, 2, flags, splits, sms)


def test_no_variant_spills():
    """A spilled register costs the step up to a tenth (fp16 with heads of 128: slower than the separate launches): its line is not in the little L1 that the kernel's shared memory leaves."""
    logs = [build.OBJ / f"step_layers_{q}.ptxas.txt" for q in ("i4", "i8", "f16")]
    if not all(p.exists() for p in logs):
        pytest.skip("the library was not built here")
    spills = re.findall(r"(\d+) bytes spill stores, (\d+) bytes spill loads", "".join(p.read_text() for p in logs))
    assert spills == [("0", "0")] * 6


def test_the_bound_of_its_waits(run, tmp_path):      # noqa: F811
    """Set for the kernel alone; the graph that holds it is captured anew."""
    path = tmp_path / "m.bin"
    binfmt.write_model(path, PLAIN, 2, binfmt.random_tensors(PLAIN, 3))
    run("""
stub.stub_sms(148)
from cuqwen_b200 import _abi
def make(flags):
    p = E.custom_params(512, 256, 512, 2, 4, 2, 64, 2, max_seq_len=256)
    p.flags = flags
    eng = E.Engine(p)
    eng.load(sys.argv[1])
    return eng
one, many = make(E.FLAG_NO_GRAPH), make(E.FLAG_NO_GRAPH | E.FLAG_NO_HANDOVER)
code = lambda e, n: _abi.lib().cuqwen_set_wait_cycles(e._h, n)
assert [code(one, n) for n in (0, 1, 2000000000, 2000000001)] == [0, 0, 0, 1] and code(many, 5) == 8
one.step(1, 0)
assert one.step_launches == 5
""", path)


def test_every_plan_is_one_that_the_kernel_can_run(built, tmp_path):
    """Alignment and sizes of copies, stages inside their slots, areas of shared memory, over the widths, head counts and SM counts that the plan takes."""
    exe = tmp_path / "probe"
    lib = build.LIB.parent
    r = subprocess.run(["g++", "-std=c++17", "-O1", f"-I{build.cuda_home() / 'include'}", str(Path(__file__).parent / "step_plan_probe.cpp"), "-o", str(exe), f"-L{lib}", "-lcuqwen_b200", f"-Wl,-rpath,{lib}",
                        f"-L{build.cuda_home() / 'lib64'}", "-lcudart"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
