"""A step whose layers are one kernel, against the oracle and against the launch-by-launch step of the same model, at the sizes where its work split, its ring
and its key ranges have their edges."""
import ctypes
import time
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from cuqwen_b200 import _abi, binfmt
from cuqwen_b200 import engine as E
from oracle import oracle_py as O
from tests.gpu_util import close, report

pytestmark = pytest.mark.gpu

MODELS = {
    # one K-part to sixteen, blocks of 8 and 40 rows, seven query heads a KV head
    "0.5b": dict(vocab=1024, dim=896, inter=4864, layers=3, heads=14, kv=2, hd=64, tied=True),
    # two q/k/v blocks in a CTA (224 on 148 SMs), the attention wider than the model, 18 key ranges a head, five query heads
    "wide attention": dict(vocab=1024, dim=256, inter=640, layers=3, heads=40, kv=8, hd=128, tied=False),
    # SwiGLU output as digits; one KV head
    "wide mlp": dict(vocab=1024, dim=256, inter=18944, layers=3, heads=8, kv=1, hd=64, tied=True),
    # the smallest: most CTAs have no work in most phases
    "one": dict(vocab=512, dim=128, inter=128, layers=1, heads=1, kv=1, hd=128, tied=True),
    # three tiles of rows a block, blocks that end beyond the matrix
    "ragged": dict(vocab=512, dim=5120, inter=1408, layers=1, heads=2, kv=2, hd=128, tied=True),
}
MAX_SEQ = 1600


def make(cfg, quant, path, flags=0, splits=0):
    p = E.custom_params(cfg["vocab"], cfg["dim"], cfg["inter"], cfg["layers"], cfg["heads"], cfg["kv"], cfg["hd"], quant, max_seq_len=MAX_SEQ)
    p.flags, p.attn_splits = flags, splits
    e = E.Engine(p)
    e.load(str(path))
    return e


def poison(eng, cfg, first):
    """NaN in every cached row from `first` on."""
    rows = np.full((MAX_SEQ - first) * cfg["hd"], np.nan, np.float16)
    for which in ("KEY_CACHE", "VALUE_CACHE"):
        base = eng.ptr(which)[0]
        for lh in range(cfg["layers"] * cfg["kv"]):
            assert _abi.lib().cuqwen_dev_upload(0, base + (lh * MAX_SEQ + first) * cfg["hd"] * 2, rows.ctypes.data_as(ctypes.c_void_p), rows.nbytes) == 0


@pytest.mark.parametrize("name", list(MODELS))
@pytest.mark.parametrize("quant", [0, 1, 2])
def test_against_the_separate_launches(built, tmp_path, name, quant):
    """Same weights, same caches, contexts around the edges of a stage (32 or 64 keys), of a key range and of sixteen stages (one key range a head).  Both steps round the same vectors
    to fp16, from sums in different orders (and the kernel does not round normalised activations of quantised weights): six vectors a layer, each off by at most half a unit in the last
    place, 2^-11 relative, of a value of its own size; over three layers the 2-norms differ by sqrt(18) / sqrt(3) x 2^-11 = 1.2e-3, of which four times is asked."""
    cfg = MODELS[name]
    path = tmp_path / "m.bin"
    binfmt.write_model(path, cfg, quant, binfmt.random_tensors(cfg, 5))
    for splits, contexts in ((0, (0, 1, 31, 32, 33, 63, 64, 65, 127, 500, 1599)), (1, (40, 513, 1200))):
        a, b = make(cfg, quant, path, 0, splits), make(cfg, quant, path, E.FLAG_NO_HANDOVER, splits)
        for ctx in contexts:
            for e in (a, b):
                e.kv_fill_normal(ctx, 7)
                poison(e, cfg, ctx)
                e.step(3 + ctx % 100, ctx)
            assert a.step_launches == 5 and b.step_launches == 1 + 6 * cfg["layers"] + 3
            la, lb = a.read("LOGITS").astype(np.float64), b.read("LOGITS").astype(np.float64)
            assert np.linalg.norm(la - lb) <= 5e-3 * np.linalg.norm(lb), (ctx, np.linalg.norm(la - lb) / np.linalg.norm(lb))
            for which in ("X", "Q", "K", "V", "ATT", "GATE"):          # what a program may read after a step
                va, vb = a.read(which).astype(np.float64), b.read(which).astype(np.float64)
                assert np.linalg.norm(va - vb) <= 5e-3 * np.linalg.norm(vb), (ctx, which)
            ka, kb = (e.read("KEY_CACHE").reshape(cfg["layers"], cfg["kv"], MAX_SEQ, cfg["hd"]) for e in (a, b))
            assert np.isfinite(ka[:, :, :ctx + 1]).all() and np.isnan(ka[:, :, ctx + 1:]).all() and close(ka[:, :, ctx], kb[:, :, ctx])
        a.close()
        b.close()


@pytest.mark.parametrize("name", ["0.5b", "wide attention"])
@pytest.mark.parametrize("quant", [0, 1, 2])
def test_against_the_oracle(built, tmp_path, name, quant):
    cfg = MODELS[name]
    path = tmp_path / "m.bin"
    binfmt.write_model(path, cfg, quant, binfmt.random_tensors(cfg, 6))
    eng, orc = make(cfg, quant, path), O.OracleModel(str(path), MAX_SEQ)
    for pos, tok in enumerate(np.random.default_rng(8).integers(0, cfg["vocab"], 36)):
        eng.step(int(tok), pos)
        orc.step(int(tok), pos)
        assert close(eng.read("LOGITS"), orc.logits), (pos, report(eng.read("LOGITS"), orc.logits))
    assert eng.step_launches == 5
    eng.close()
    orc.close()


@pytest.mark.parametrize("name", ["0.5b", "wide attention"])
@pytest.mark.parametrize("quant", [0, 1, 2])
def test_long_contexts_against_the_oracle(built, tmp_path, name, quant):
    """The last context of one key range a KV head, and several ranges (18 or 74 at most), whose partials travel between CTAs and are merged: the oracle goes on from the engine's own filled cache."""
    cfg = MODELS[name]
    path = tmp_path / "m.bin"
    binfmt.write_model(path, cfg, quant, binfmt.random_tensors(cfg, 6))
    eng, orc = make(cfg, quant, path), O.OracleModel(str(path), MAX_SEQ)
    shape = (cfg["layers"], cfg["kv"], MAX_SEQ, cfg["hd"])
    eng.kv_fill_normal(MAX_SEQ, 7)
    for view, which in zip(orc.kv_views(), ("KEY_CACHE", "VALUE_CACHE")):
        view[...] = eng.read(which).reshape(shape)
    for ctx in (255, 256, 700, 1599):
        eng.step(3 + ctx % 100, ctx)
        orc.step(3 + ctx % 100, ctx)
        assert close(eng.read("LOGITS"), orc.logits), (ctx, report(eng.read("LOGITS"), orc.logits))
        for view, which in zip(orc.kv_views(), ("KEY_CACHE", "VALUE_CACHE")):
            got = eng.read(which).reshape(shape)[:, :, ctx]
            assert close(got, view[:, :, ctx]), (ctx, which, report(got, view[:, :, ctx]))
            view[:, :, ctx] = got                      # each step over the same cache
    assert eng.step_launches == 5
    eng.close()
    orc.close()


def test_steps_of_two_engines_do_not_mix(built, tmp_path):
    """Their exchange words are their own, and a step's numbers go on when the control block is written anew (decode_n, a profile, which runs the separate launches)."""
    cfg = MODELS["0.5b"]
    path = tmp_path / "m.bin"
    binfmt.write_model(path, cfg, 2, binfmt.random_tensors(cfg, 9))
    a, b, c = (make(cfg, 2, path) for _ in range(3))
    want = [a.step(5, 0)]
    for i in range(1, 24):
        want.append(a.step(want[-1], i))
    got = b.decode_n(5, 0, 8).tolist()
    b.profile_step(got[-1], 8)
    other = c.step(9, 0)
    for i in range(8, 16):
        got.append(b.step(got[-1], i))
        other = c.step(other, i - 7)
    got += b.decode_n(got[-1], 16, 8).tolist()
    assert got == want
    for e in (a, b, c):
        e.close()


@pytest.mark.parametrize("flags", [0, E.FLAG_SEPARATE_KERNELS])
def test_engines_in_several_threads(built, tmp_path, flags):
    """A step's kernel takes the whole GPU, all of it at once: engines that are called from several threads go one step at a time, or share it kernel by kernel, and each gets what it gets alone."""
    cfg = MODELS["0.5b"]
    path = tmp_path / "m.bin"
    binfmt.write_model(path, cfg, 2, binfmt.random_tensors(cfg, 9))

    def tokens(e, first):
        out = [e.step(first, 0)]
        for i in range(1, 60):
            out.append(e.step(out[-1], i))
        return out + e.decode_n(out[-1], 60, 100).tolist() + e.step_loop(7, 160, 60).tolist()

    engines = [make(cfg, 2, path, flags) for _ in range(3)]
    alone = [tokens(e, 5 + i) for i, e in enumerate(engines)]
    assert {e.step_launches for e in engines} == {1 + 6 * cfg["layers"] + 3 if flags else 5}
    with ThreadPoolExecutor(len(engines)) as ex:
        assert list(ex.map(tokens, engines, range(5, 8))) == alone
    for e in engines:
        e.close()


@pytest.mark.parametrize("quant,heads,kv,hd,ctx", [(2, 28, 4, 128, 1500), (2, 14, 2, 64, 250), (0, 14, 2, 64, 1500)])
def test_the_same_step_again(built, tmp_path, quant, heads, kv, hd, ctx):
    """Every sum of a step has one order, so that a step repeated over the same caches gives the same bits, however the CTAs happen to run: many heads, whose attention is merged and staged
    at different times, and one range a KV head."""
    cfg = dict(vocab=512, dim=512, inter=1024, layers=4, heads=heads, kv=kv, hd=hd, tied=True)
    path = tmp_path / "m.bin"
    binfmt.write_model(path, cfg, quant, binfmt.random_tensors(cfg, 5))
    e = make(cfg, quant, path)
    e.kv_fill_normal(ctx, 7)
    e.step(5, ctx)
    assert e.step_launches == 5
    first = e.read("LOGITS")
    for i in range(1000):
        e.step(5, ctx)
        assert np.array_equal(e.read("LOGITS").view(np.uint16), first.view(np.uint16)), i
    e.close()


@pytest.mark.parametrize("dim,inter,heads,kv,hd", [(896, 4864, 14, 2, 64), (1536, 8960, 12, 2, 128), (2048, 11008, 16, 2, 128)])
@pytest.mark.parametrize("quant", [0, 1, 2])
def test_steps_at_changing_places(built, tmp_path, quant, dim, inter, heads, kv, hd):
    """What a CTA prepares before the first layer, the rotation and its rows of the residual stream, is the step's own: tokens and positions that jump from step to step, up to 256 keys (many CTAs
    begin with the output projection) and beyond.  Layer 0's key row and the logits are those of the separate launches (bound: see above), and a step's bits do not depend on the step before
    it (each runs over the same cached rows in both orders)."""
    cfg = dict(vocab=512, dim=dim, inter=inter, layers=2, heads=heads, kv=kv, hd=hd, tied=True)
    path = tmp_path / "m.bin"
    binfmt.write_model(path, cfg, quant, binfmt.random_tensors(cfg, 5))
    a, b = make(cfg, quant, path), make(cfg, quant, path, E.FLAG_NO_HANDOVER)
    rng = np.random.default_rng(3)
    places = [(int(rng.integers(512)), int(rng.integers(*r))) for _ in range(20) for r in ((0, 256), (256, MAX_SEQ))]

    def run(e, tok, pos):
        e.kv_fill_normal(pos, 7)
        e.step(tok, pos)
        return e.read("LOGITS"), e.read("KEY_CACHE").reshape(2, kv, MAX_SEQ, hd)[0, :, pos]

    first = [run(a, *p) for p in places]
    assert a.step_launches == 5
    for p, got in zip(places, first):
        for g, w in zip(got, run(b, *p)):
            g, w = g.astype(np.float64), w.astype(np.float64)
            assert np.linalg.norm(g - w) <= 5e-3 * np.linalg.norm(w), p
    for i in np.random.default_rng(4).permutation(len(places)):
        for g, w in zip(run(a, *places[i]), first[i]):
            assert np.array_equal(g.view(np.uint16), w.view(np.uint16)), places[i]
    a.close()
    b.close()


@pytest.mark.parametrize("quant,hd", [(2, 64), (1, 128), (0, 128)])
@pytest.mark.parametrize("cycles", [1, 20000])
def test_waits_that_expire(built, tmp_path, quant, hd, cycles):
    """Waits that end before the words and copies that they are for are there (at their first look; in the middle of the step, which takes some 100,000 cycles): the step, also one that feeds itself,
    ends with an error and in time, and the next one, with waits of the usual length, is the same as an undisturbed engine's."""
    cfg = dict(vocab=512, dim=512, inter=1024, layers=6, heads=4, kv=2, hd=hd, tied=True)
    path = tmp_path / "m.bin"
    binfmt.write_model(path, cfg, quant, binfmt.random_tensors(cfg, 5))
    e, whole = make(cfg, quant, path), make(cfg, quant, path)
    for ctx in (40, 1200):
        whole.kv_fill_normal(ctx, 7)
        whole.step(5, ctx)
        _abi.check(_abi.lib().cuqwen_set_wait_cycles(e._h, cycles))
        for _ in range(3):
            e.kv_fill_normal(ctx, 7)
            begin = time.perf_counter()
            for call in (lambda: e.step(5, ctx), lambda: e.decode_n(5, ctx, 4)):
                with pytest.raises(_abi.CuQwenError) as err:
                    call()
                assert err.value.code == 9
            assert time.perf_counter() - begin < 5
        _abi.check(_abi.lib().cuqwen_set_wait_cycles(e._h, 0))
        e.kv_fill_normal(ctx, 7)
        e.step(5, ctx)
        for which in ("LOGITS", "KEY_CACHE"):
            got, want = (x.read(which).reshape(-1) if which == "LOGITS" else x.read(which).reshape(6, 2, MAX_SEQ, hd)[:, :, :ctx + 1] for x in (e, whole))
            assert np.array_equal(got.view(np.uint16), want.view(np.uint16)), which
    e.close()
    whole.close()
