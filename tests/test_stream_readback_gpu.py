"""Read-back entries right after the prompts of an engine of several streams: the prompt passes are wider than the cycles, a
row is still row r % (k + 1) of stream r / (k + 1)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _f(u):
    return np.array(u, dtype=np.uint32).view(np.float32)


@pytest.mark.parametrize("d,quant", [(256, "q8_0"), (2304, "q4_k_m")])   # (a wide Q6_K head's K-split differs between the two widths)
@pytest.mark.parametrize("B,k,drafter", [(2, 0, False), (4, 1, False), (4, 1, True), (1, 0, False)])
def test_rows_of_the_last_prompt_pass(pkg, packs, oracle, llb, B, k, drafter, d, quant):
    cfg = packs.cfg_tiny(d_model=d, quant=quant, tied_head=False, seed=23)
    pack = packs.build_pack(cfg)
    mtp = packs.aux1_bytes(packs.build_mtp(pack)) if drafter else None
    prompts = [packs.synth_prompt(b, 14 + 3 * b, cfg.vocab_size) for b in range(B)]
    eng = pkg.llb.SpecEngine(pack, mtp, k=k, max_ctx=96, streams=B)
    one = pkg.llb.SpecEngine(pack, mtp, k=k, max_ctx=96)
    try:
        if B > 1:
            eng.prefill_streams(prompts)
        else:
            eng.prefill(prompts[0])
        for b, p in enumerate(prompts):
            # the last prompt pass of a stream has at most k + 1 rows; its last one is the position before the prompt's last token
            n = len(p) - 1
            width = 16 // B if B > 1 else 8
            rest = n
            while rest > k + 1:
                rest -= min(rest - (k + 1), width)
            lg = eng.read_logits(b * (k + 1) + rest - 1)
            orc = oracle.Oracle(pack.index_text(), pack.data.numpy(), cap=64)
            _ids, top2 = orc.greedy(p[:-1], 1)
            orc.close()
            ref_id, ref_v, gap = int(top2[0][0]), float(_f(top2[0][1])), float(_f(top2[0][1]) - _f(top2[0][3]))
            assert abs(lg[ref_id] - ref_v) <= 2e-2 + 1e-2 * abs(ref_v)
            assert int(lg.argmax()) == ref_id or gap < 1e-3
            one.prefill(p)
            hn = eng.read_state_stream(b, 4, 0, rest - 1) if B > 1 else eng.read_state(4, 0, rest - 1)
            ref = one.read_state(4, 0, rest - 1)
            assert np.abs(ref).max() > 0 and np.abs(hn - ref).max() <= 2e-2 + 1e-2 * np.abs(ref).max()
    finally:
        eng.close()
        one.close()
