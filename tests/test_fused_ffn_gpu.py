"""The one-launch FFN (llb_b200_use_fused_ffn) at the widths where its shared memory decides: gate|up's planes of all d columns
beside the ring, with each format of the down matrix.  Where it runs, the pass has fewer kernels; ids equal the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
STEPS = 12


def _f(u):
    return np.array(u, dtype=np.uint32).view(np.float32)


# 6656 columns are the most that fit; the last one runs as three launches
@pytest.mark.parametrize("d,f,down,runs", [(3840, 1024, "Q6_K", True), (5120, 1024, "Q4_K", True), (6656, 512, "Q5_K", True), (256, 76800, "Q5_K", True), (6912, 512, "Q4_K", False)])
def test_fused_ffn_widths(pkg, packs, oracle, llb, monkeypatch, d, f, down, runs):
    L = llb.lib()
    monkeypatch.setenv("LLB_PREFILL_ROWS", "4")   # (76800 columns do not fit eight-row prompt passes)
    cfg = packs.cfg_tiny(quant="q4_k_m", n_layers=4, d_model=d, d_ff=f, seed=14, type_overrides=(("ffn_down", down),))
    pack = packs.build_pack(cfg)
    prompt = packs.synth_prompt(5, 7, cfg.vocab_size)
    orc = oracle.Oracle(pack.index_text(), pack.data.numpy(), cap=40)
    ref_ids, ref_top2 = orc.greedy(prompt, STEPS)
    orc.close()
    nodes = {}
    for on in (0, 1):
        was = L.llb_b200_use_fused_ffn(on)
        try:
            eng = pkg.llb.SpecEngine(pack, None, k=0, max_ctx=40)
            nodes[on] = eng.graph_nodes(2)
            eng.prefill(prompt)
            ids, top2 = eng.generate(STEPS)
            eng.close()
        finally:
            L.llb_b200_use_fused_ffn(was)
        same = STEPS
        for i in range(STEPS):
            if ids[i] != ref_ids[i]:
                gap = float(_f(ref_top2[i][1]) - _f(ref_top2[i][3]))
                assert gap < 1e-3, f"token {i}: device {ids[i]}, oracle {ref_ids[i]}, oracle top-2 gap {gap}"
                same = i
                break
        v, r = _f(top2[:same, 1]), _f(ref_top2[:same, 1])
        assert np.all(np.abs(v - r) <= 2e-2 + 1e-2 * np.abs(r)), float(np.abs(v - r).max())
    assert L.llb_b200_wait_errors() == 0
    assert (nodes[1] < nodes[0]) == runs
