"""Prompts in mode 0 (llb_spec_set_prefill(0)): more than four rows (and k + 1) go through the dense path's exact forms in pieces of 128 rows, whole, without a
T-row pass behind them.  Against T-row passes (LLB_PREFILL_ROWS) on the same model: state, K/V rows, the rows left for the drafter, logits of
the last prompt row, ids; the same bits whatever k is and whether several streams' prompts are fed together or in turn."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
STEPS = 12


def _f(u):
    return np.ascontiguousarray(np.array(u, dtype=np.uint32)).view(np.float32)


def _run(pkg, pack, mtp, k, prompt, last):
    cfg = pack.cfg
    eng = pkg.llb.SpecEngine(pack, mtp if k else None, k=k, max_ctx=len(prompt) + STEPS * (k + 1) + 24)
    try:
        eng.prefill(prompt)
        n = len(prompt)
        st = {}
        for il in range(cfg.n_layers):
            if cfg.is_full(il):
                for what in (1, 2):
                    st[f"kv{what}.{il}"] = np.stack([eng.read_state(what, il, p) for p in (0, n // 2, n - 2)])
            else:
                st[f"S{il}"] = eng.read_state(0, il)
                st[f"c{il}"] = np.stack([eng.read_state(3, il, p) for p in range(max(0, n - 4), n - 1)])
        if k:
            st["mk"] = np.stack([eng.read_state(5, 0, p) for p in (0, n // 2, n - 1 - (k + 1), n - 2)])   # the last k + 1 are left to the drafter
        st["hn"] = np.stack([eng.read_state(4, 0, r) for r in range(last)])
        st["lg"] = eng.read_logits(last - 1)
        ids, t2 = eng.generate(STEPS)
        assert eng.fast_rows() == 0 and pkg.llb.lib().llb_b200_wait_errors() == 0
        return st, ids, t2
    finally:
        eng.close()


@pytest.mark.parametrize("n", [5, 6, 9, 18, 41, 129, 130, 136, 137, 138, 260])   # rows at the edges of the rule, of units and of pieces (a last one under eight rows is not cut)
def test_pieces_against_t_row_passes(pkg, packs, llb, monkeypatch, n):
    pack = packs.build_pack(packs.cfg_tiny(n_layers=4, seed=31, quant="q4_k_m"))
    mtp = packs.aux1_bytes(packs.build_mtp(pack))
    prompt = packs.synth_prompt(n, n, pack.cfg.vocab_size)
    runs = {k: _run(pkg, pack, mtp, k, prompt, k + 1) for k in (0, 3)}
    assert np.array_equal(runs[0][1], runs[3][1]) and np.array_equal(runs[0][2], runs[3][2])     # lossless, bit for bit
    for key, v in runs[0][0].items():
        if key not in ("hn", "lg"):
            assert np.array_equal(v.view(np.uint32), runs[3][0][key].view(np.uint32)), key
    monkeypatch.setenv("LLB_PREFILL_ROWS", "8")
    st, ids, t2 = _run(pkg, pack, mtp, 3, prompt, 4)
    for key, v in st.items():    # sums in another order, amplified by four layers: far inside the path's bars
        assert np.all(np.abs(v - runs[3][0][key]) <= 2e-4 + 1e-3 * np.abs(v)), (key, float(np.abs(v - runs[3][0][key]).max()))
    for i in range(STEPS):
        if ids[i] != runs[3][1][i]:
            assert _f(t2[i])[1] - _f(t2[i])[3] < 1e-3, i
            break


@pytest.mark.parametrize("k", [4, 7])
def test_prompts_that_one_t_row_pass_takes(pkg, packs, llb, monkeypatch, k):
    """With k >= 4 a prompt of five to k + 1 rows is one T-row pass and stays that; one row more takes the dense path, as with any k."""
    pack = packs.build_pack(packs.cfg_tiny(n_layers=4, seed=34, quant="q4_k_m"))
    mtp = packs.aux1_bytes(packs.build_mtp(pack))

    def state(kk, rows):
        eng = pkg.llb.SpecEngine(pack, mtp, k=kk, max_ctx=96)
        try:
            eng.prefill(packs.synth_prompt(rows, rows + 1, pack.cfg.vocab_size))
            return np.concatenate([eng.read_state(0, il) for il in range(pack.cfg.n_layers) if not pack.cfg.is_full(il)]).view(np.uint32)
        finally:
            eng.close()

    one, more, dense = state(k, k + 1), state(k, k + 2), state(3, k + 2)
    assert np.array_equal(more, dense)
    assert not np.array_equal(one, state(3, k + 1))
    monkeypatch.setenv("LLB_PREFILL_ROWS", "8")
    assert np.array_equal(one, state(k, k + 1))
    assert not np.array_equal(more, state(k, k + 2))


def test_streams_together_and_in_turn(pkg, packs, llb):
    """Five prompts: two of several pieces, three that share a chunk with others, one in T-row passes, one of a single token."""
    pack = packs.build_pack(packs.cfg_tiny(n_layers=4, seed=32))
    mtp = packs.aux1_bytes(packs.build_mtp(pack))
    lens = [40, 150, 5, 1, 261]
    prompts = [packs.synth_prompt(200 + b, n, pack.cfg.vocab_size) for b, n in enumerate(lens)]
    out = []
    for together in (False, True):
        eng = pkg.llb.SpecEngine(pack, mtp, k=2, max_ctx=320, streams=5)
        try:
            if together:
                eng.prefill_streams(prompts)
            else:
                for b, p in enumerate(prompts):
                    eng.prefill_stream(b, p)
            states = [eng.read_state_stream(b, 0, 0) for b in range(5)]
            got = [[] for _ in prompts]
            for _ in range(6):
                for b, (i, t) in enumerate(eng.cycle_streams()):
                    got[b] += [(int(v), tuple(int(x) for x in r)) for v, r in zip(i, t)]
            out.append((got, states))
        finally:
            eng.close()
    assert out[0][0] == out[1][0]
    for a, b in zip(out[0][1], out[1][1]):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))


@pytest.mark.parametrize("streams", [1, 3])
def test_nothing_is_left_to_the_next_call(pkg, packs, llb, streams):
    """The library's stream is idle when a prompt's call returns, the pass over its last rows' logits included (a head that takes a while)."""
    import torch
    pack = packs.build_pack(packs.cfg_tiny(n_layers=4, seed=33, vocab_size=200000))
    eng = pkg.llb.SpecEngine(pack, None, k=0, max_ctx=96, streams=streams)
    try:
        stream = torch.cuda.ExternalStream(pkg.llb.lib().llb_b200_stream())
        prompts = [packs.synth_prompt(300 + b, 40, pack.cfg.vocab_size) for b in range(streams)]
        for _ in range(5):
            eng.prefill_streams(prompts) if streams > 1 else eng.prefill(prompts[0])
            assert stream.query()
    finally:
        eng.close()
