"""Which kernels a call launches, on the CPU over tests/cudart_stub.cpp."""
import pytest

from cuqwen_b200 import binfmt
from gemm_plans import PLANS
from test_host_memory import run                                           # noqa: F401  (fixture)


@pytest.mark.parametrize("hd,sms,sizes", [
    # (tokens, position) -> the mma.sync kernel, else the tcgen05 one; two heads
    (128, 148, [(1, 0, True), (512, 0, True), (513, 0, False), (100, 412, True), (100, 413, False), (1, 9000, False)]),
    (64, 148, [(1, 0, True), (4736, 0, True), (4737, 0, False), (64, 9000, True)]),
    (64, 7, [(192, 0, True), (193, 0, False), (64, 9000, True)]),
])
def test_attention_kernel_of_a_prompt(run, tmp_path, hd, sms, sizes):      # noqa: F811
    cfg = dict(vocab=512, dim=256, inter=512, layers=2, heads=2, kv=1, hd=hd, tied=True)
    path = tmp_path / "m.bin"
    binfmt.write_model(path, cfg, 2, binfmt.random_tensors(cfg, 3))
    run(f"""
stub.stub_sms({sms})
eng = E.Engine(E.custom_params(512, 256, 512, 2, 2, 1, {hd}, 2, max_seq_len=10000))
eng.load(sys.argv[1])
for n, pos, mma in {sizes}:
    stub.stub_launches()
    eng.prefill(toks[:n], pos)
    names = stub.stub_launches().decode()
    assert ("prefill_attn_kernel" in names, "prefill_attn_tc_kernel" in names) == (mma, not mma), (n, pos, names)
""", path)


def test_blocks_of_a_decode_product(run):                                  # noqa: F811
    """CTAs of a GEMV: blocks that end in one round where that was measured to pay, whole tiles (then every SM has a CTA) elsewhere."""
    run("""
from cuqwen_b200 import kernels as K
def grid(quant, rows, cols, gate_up):
    stub.stub_launches()
    s = 4096 if quant else None
    if gate_up: K.fused_mlp_stage1(quant, 4096, 4096, 4096, s, s, 4096, cols, rows)
    else: K.gemv_add(quant, 4096, s, 4096, 4096, rows, cols)
    name, grid, _ = stub.stub_launches().decode().split()
    assert "gemv_kernel" in name
    return int(grid.split(",")[0])
for quant, rows, cols, gate_up, ctas in [(1, 7168, 896, False, 128), (1, 4864, 896, True, 122), (2, 4864, 896, True, 122), (2, 11008, 2048, True, 138),      # blocks below 100 KB, int4
                                         (0, 5120, 3584, False, 128), (1, 11008, 2048, True, 138), (0, 6912, 3584, False, 148), (1, 8192, 3584, True, 148),   # about a ring
                                         (0, 27648, 896, False, 148), (1, 13824, 1536, True, 148),
                                         (1, 13824, 5120, True, 144), (0, 13824, 3584, False, 144), (0, 8192, 5120, False, 148)]:                            # several rings
    assert grid(quant, rows, cols, gate_up) == ctas, (quant, rows, cols, gate_up, grid(quant, rows, cols, gate_up), ctas)
""")


PLAN_OF = """
import re
from cuqwen_b200 import binfmt
from cuqwen_b200 import kernels as K
def plan(quant, kind, tokens, rows, cols):
    stub.stub_launches()
    s = 4096 if quant else None
    if quant == 3: K.linear(0, K.LIN_F32, 4096, cols, 4096, -(-cols // 128) * 128, cols, tokens, rows, 4096, rows)
    elif kind == "swiglu": K.prefill_gemm(quant, K.PF_SWIGLU, 4096, 4096, s, 4096, tokens, rows, cols, w1=4096, s1=s)
    else: K.prefill_gemm(quant, K.PF_RESID, 4096, 4096, s, 4096, tokens, rows, cols)
    name, _, cluster = stub.stub_launches().decode().split()
    return tuple(int(v) for v in re.search("prefill_gemm_kernelILi.ELi(\\d+)ELi(\\d+)ELi(\\d+)E", name).groups()) + (int(cluster.split(",")[2]),)
"""


def test_products_stand_under_the_plan_they_take(run):                     # noqa: F811
    run(PLAN_OF + f"""
for (quant, kind), sizes in {PLANS}.items():
    for want, size in sizes.items():
        assert plan(quant, kind, *size) == want, (quant, kind, size, want, plan(quant, kind, *size))
""")


def test_no_model_takes_a_plan_that_is_not_tested(run):                    # noqa: F811
    """The products of the table's models and of the designs' two sizes, at token counts over the whole range of a portion."""
    designs = [(1536, 13440), (13440, 1536), (1536, 1536), (576, 1536), (6400, 1536), (1536, 6400), (8064, 1536), (64, 1536), (3584, 25600), (25600, 3584), (3584, 3584),
               (12928, 3584), (3584, 12928), (1024, 3584), (16896, 3584)]
    run(PLAN_OF + f"""
tested = {PLANS}
tokens = sorted(set(list(range(1, 300, 13)) + [int(1.11 ** i) for i in range(1, 87)] + [128, 129, 256, 257, 512, 513, 8192]))
for n in tokens:
    for m in binfmt.MODELS.values():
        for quant in (0, 1, 2):
            for kind, rows, cols in (("plain", (m["heads"] + 2 * m["kv"]) * m["hd"], m["dim"]), ("plain", m["dim"], m["heads"] * m["hd"]), ("swiglu", m["inter"], m["dim"]), ("plain", m["dim"], m["inter"])):
                assert plan(quant, kind, n, rows, cols) in tested[quant, kind], (quant, kind, n, rows, cols)
    for rows, cols in {designs}:
        if 2 <= n <= 4096:
            assert plan(3, "plain", n, rows, cols) in tested[3, "plain"], (n, rows, cols)
""")


def test_a_plan_on_any_number_of_sms(run):                                 # noqa: F811
    """Down to one SM, of which no cluster of four fits any."""
    run(PLAN_OF + """
for sms in (0, 1, 2, 3, 7, 20, 74, 132, 148, 160):
    stub.stub_sms(sms)
    for size in ((5, 72, 2048), (61, 896, 4864), (700, 6408, 256), (4096, 1536, 1536)):
        for quant in range(4):
            assert plan(quant, "plain", *size)[0] in (64, 128, 192, 224, 256)
""")
