"""The prompt path's buffers belong to the engine that has the weights and serve all of its siblings: prompts of several engines at once from
threads, the first ones included, and prompts between another engine's prompt and cycles, leave what each leaves alone."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STEPS = 6
LENS = [300, 40, 150, 9]


@pytest.fixture(scope="module")
def model(pkg, packs, llb):
    pack = packs.build_pack(packs.cfg_tiny(n_layers=4, seed=61))
    return pack, packs.aux1_bytes(packs.build_mtp(pack))


def _open(pkg, model, n):
    first = pkg.llb.SpecEngine(model[0], model[1], k=3, max_ctx=360)
    return [first] + [first.sibling(k=i % 4, max_ctx=360) for i in range(n - 1)]


def _result(eng, cfg):
    st = [eng.read_state(0, il) for il in range(cfg.n_layers) if not cfg.is_full(il)] + [eng.read_state(4, 0, 0)]
    return st, eng.generate(STEPS)


def _same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a[0], b[0])) and all(np.array_equal(x, y) for x, y in zip(a[1], b[1]))


def _at_once(calls):
    gate, errors = threading.Barrier(len(calls)), []

    def run(call):
        try:
            gate.wait()
            call()
        except Exception as e:   # noqa: BLE001 - any failure of a thread is the test's
            errors.append(repr(e))

    ts = [threading.Thread(target=run, args=(c,)) for c in calls]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors


@pytest.mark.parametrize("fast", [False, True])
def test_first_prompts_at_once(pkg, packs, model, fast):
    cfg = model[0].cfg
    prompts = [packs.synth_prompt(70 + i, n, cfg.vocab_size) for i, n in enumerate(LENS)]
    want = []
    for i, p in enumerate(prompts):
        engs = _open(pkg, model, len(prompts))
        engs[i].set_prefill(fast)
        engs[i].prefill(p)
        want.append(_result(engs[i], cfg))
        for e in engs:
            e.close()
    for _ in range(3):
        engs = _open(pkg, model, len(prompts))
        for e in engs:
            e.set_prefill(fast)
        _at_once([lambda e=e, p=p: e.prefill(p) for e, p in zip(engs, prompts)])
        for e, w in zip(engs, want):
            assert _same(_result(e, cfg), w)
        for e in engs:
            e.close()


def test_prompt_between_another_ones_prompt_and_cycles(pkg, packs, model):
    cfg = model[0].cfg
    a, b = (packs.synth_prompt(90 + i, n, cfg.vocab_size) for i, n in enumerate((290, 133)))
    engs = _open(pkg, model, 2)
    engs[0].prefill(a)
    want = _result(engs[0], cfg)
    engs[0].prefill(a)
    engs[1].prefill(b)
    assert _same(_result(engs[0], cfg), want)
    engs[1].prefill(b)
    other = _result(engs[1], cfg)
    engs[1].prefill(b)
    engs[0].prefill(a)
    assert _same(_result(engs[1], cfg), other)
    for e in engs:
        e.close()


def test_no_room(pkg, packs, model, monkeypatch):
    """No room for the prompt path's buffers: a default prompt goes through T-row passes, one of mode 1 is refused; once there is room both take them."""
    cfg, L = model[0].cfg, pkg.llb.lib()
    p = packs.synth_prompt(80, 140, cfg.vocab_size)

    def alone(fast):
        eng = pkg.llb.SpecEngine(model[0], model[1], k=3, max_ctx=200)
        eng.set_prefill(fast)
        eng.prefill(p)
        r = _result(eng, cfg)
        eng.close()
        return r

    want = [alone(False), alone(True)]
    monkeypatch.setenv("LLB_PREFILL_ROWS", "8")
    t_rows = alone(False)
    monkeypatch.delenv("LLB_PREFILL_ROWS")
    assert not _same(t_rows, want[0])      # (sums in another order: which path a prompt took shows)
    engs = _open(pkg, model, 2)
    engs[1].close()
    first, sib = engs[0], engs[0].sibling(k=3, max_ctx=200)
    for _ in range(2):
        L.llb_spec_prefill_extra(first.h, 1 << 50)
        for e in (first, sib):
            e.set_prefill(False)
            e.prefill(p)
            assert _same(_result(e, cfg), t_rows)
            e.set_prefill(True)
            with pytest.raises(Exception, match="buffers take"):
                e.prefill(p)
    L.llb_spec_prefill_extra(sib.h, 0)
    for fast in (False, True):
        for e in (sib, first):
            e.set_prefill(fast)
            e.prefill(p)
            assert _same(_result(e, cfg), want[fast])
    sib.close()
    first.close()


def test_rows_of_the_last_chunk(pkg, packs, model):
    """read_state of kind 6: a stream's own rows of a chunk that several streams share, and nothing once a sibling's chunk came after it."""
    cfg = model[0].cfg
    first = pkg.llb.SpecEngine(model[0], model[1], k=3, max_ctx=360)
    eng, lens = first.sibling(k=3, max_ctx=360, streams=3), (41, 31, 21)
    eng.prefill_streams([packs.synth_prompt(50 + b, n, cfg.vocab_size) for b, n in enumerate(lens)])
    for b, n in enumerate(lens):
        for r in range(4):          # the rows left for the drafter are the piece's last
            assert np.array_equal(eng.read_state_stream(b, 6, 0, n - 1 - 4 + r), eng.read_state_stream(b, 4, 0, r)), (b, r)
        with pytest.raises(Exception, match="no row"):
            eng.read_state_stream(b, 6, 0, n - 1)
    first.prefill(packs.synth_prompt(55, 150, cfg.vocab_size))
    with pytest.raises(Exception, match="no row"):
        eng.read_state_stream(0, 6, 0, 0)
    assert np.array_equal(first.read_state(6, 0, 149 - 128 - 1), first.read_state(4, 0, 3))
    eng.close()
    first.close()


def test_engines_of_different_streams_at_once(pkg, packs, model):
    """One engine feeds the prompts of three streams, others one each, from threads: nobody enqueues with another one's stream geometry."""
    cfg = model[0].cfg
    first = pkg.llb.SpecEngine(model[0], model[1], k=3, max_ctx=360)
    many, other = first.sibling(k=3, max_ctx=360, streams=3), first.sibling(k=0, max_ctx=360)
    three = [packs.synth_prompt(30 + b, n, cfg.vocab_size) for b, n in enumerate((150, 40, 30))]
    ones = [packs.synth_prompt(35 + b, 60 + b, cfg.vocab_size) for b in range(2)]

    def three_result():
        return [many.read_state_stream(b, 0, 0) for b in range(3)], [many.cycle_streams() for _ in range(3)]

    def same(a, b):
        return all(np.array_equal(x, y) for x, y in zip(a[0], b[0])) and all(
            np.array_equal(i, j) and np.array_equal(t, u) for x, y in zip(a[1], b[1]) for (i, t), (j, u) in zip(x, y))

    many.prefill_streams(three)
    want = [three_result()]
    for e, p in zip((first, other), ones):
        e.prefill(p)
        want.append(_result(e, cfg))
    for _ in range(5):
        _at_once([lambda: many.prefill_streams(three), lambda: first.prefill(ones[0]), lambda: other.prefill(ones[1])])
        assert same(three_result(), want[0])
        assert _same(_result(first, cfg), want[1]) and _same(_result(other, cfg), want[2])
    for e in (many, other, first):
        e.close()
