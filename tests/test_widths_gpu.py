"""Widths at which the usual rings of weight tiles leave a K-slice of activations no room in shared memory: one K-slice of
wide routed-expert models, matrices of more than sixteen of the usual slices, and several streams whose wide prompt passes
need more of it than their cycles."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _f(u):
    return np.array(u, dtype=np.uint32).view(np.float32)


# super-blocks that a slice holds beside the usual ring and beside the shorter one: Q4_K 17 and 26 at 8 plane columns (up to
# four rows), 8 and 13 at 16; Q6_K 8 and 11 at 32
@pytest.mark.parametrize("d,rows,B,ty", [(2304, 8, 1, "Q4_K"), (3072, 8, 1, "Q4_K"), (4608, 4, 1, "Q4_K"), (6400, 4, 1, "Q4_K"), (2304, 1, 16, "Q6_K")])
def test_wide_expert_models(pkg, packs, oracle, llb, monkeypatch, d, rows, B, ty):
    cfg = packs.cfg_tiny_moe(n_layers=2, d_model=d, type_overrides=(("ffn_gate", ty), ("ffn_up", ty)))
    pack = packs.build_pack(cfg)
    monkeypatch.setenv("LLB_PREFILL_ROWS", str(rows))
    T = rows * B
    h2 = np.random.default_rng(d).standard_normal((T, d), dtype=np.float32)
    eng = pkg.llb.SpecEngine(pack, None, k=rows - 1, max_ctx=64, streams=B)
    orc = oracle.Oracle(pack.index_text(), pack.data.numpy(), cap=8)
    try:
        out, ids, wt = eng.moe_ffn(1, h2)
        for t in range(T):
            ro, rid, rw = orc.moe_ffn(1, h2[t])
            assert list(ids[t, :cfg.n_experts_used]) == list(rid[:cfg.n_experts_used])
            assert np.linalg.norm(out[t] - ro) / np.linalg.norm(ro) < 2e-5
        assert llb.lib().llb_b200_wait_errors() == 0
    finally:
        eng.close()
        orc.close()


def test_streams_of_a_wide_expert_model(pkg, packs, oracle, llb):
    """Two streams of plain decoding: their passes have two rows (8 plane columns), sixteen rows a prompt pass would not fit."""
    cfg = packs.cfg_tiny_moe(n_layers=4, d_model=3072)
    pack = packs.build_pack(cfg)
    prompts = [packs.synth_prompt(b, 11 + 4 * b, cfg.vocab_size) for b in range(2)]
    eng = pkg.llb.SpecEngine(pack, None, k=0, max_ctx=64, streams=2)
    try:
        eng.prefill_streams(prompts)
        got = [[] for _ in prompts]
        for _ in range(12):
            for b, (i, _t) in enumerate(eng.cycle_streams()):
                got[b] += [int(v) for v in i]
    finally:
        eng.close()
    for b, p in enumerate(prompts):
        orc = oracle.Oracle(pack.index_text(), pack.data.numpy(), cap=64)
        ref, top2 = orc.greedy(p, 12)
        orc.close()
        for i in range(12):
            if got[b][i] != ref[i]:
                gap = float(_f(top2[i][1]) - _f(top2[i][3]))
                assert gap < 1e-3, f"stream {b} token {i}: device {got[b][i]}, oracle {ref[i]}, oracle top-2 gap {gap}"
                break


@pytest.mark.parametrize("K,T", [(256 * 129, 8), (256 * 192, 5), (256 * 273, 1), (256 * 400, 4)])
def test_more_columns_than_sixteen_usual_slices(llb, packs, dev, K, T):
    rng = np.random.default_rng(K)
    rows, ty, L = 40, "Q4_K", llb.lib()
    raw = packs.QUANT[ty](torch.from_numpy(rng.standard_normal((rows, K), dtype=np.float32) * 0.05))
    x = rng.standard_normal((T, K), dtype=np.float32)
    w = dev(L.llb_b200_weight_bytes(packs.FMT[ty], rows, K))
    llb.check(L.llb_b200_weight_upload(packs.FMT[ty], rows, K, raw.numpy().ctypes.data, 0, w.ptr), "weight_upload")
    xd, y = dev(x.nbytes).write(x), dev(T * rows * 4)
    xp = llb.handle(L.llb_b200_xp_new(K, T, 2), "xp_new")
    llb.check(L.llb_b200_xp_set_f32(xp, xd.ptr), "xp_set")
    llb.gemm(packs.FMT[ty], [w.ptr], [rows], [y.ptr], K, xp, 0)
    got = y.read((T, rows), np.float32)
    L.llb_b200_xp_free(xp)
    deq = packs.dequant(ty, raw, rows, K).numpy().astype(np.float64)
    # activations to about 22 bits, f32 sums: 1e-5 of the sum of the products' magnitudes
    assert np.all(np.abs(got - x.astype(np.float64) @ deq.T) <= 1e-5 * (np.abs(x).astype(np.float64) @ np.abs(deq).T))
    assert L.llb_b200_wait_errors() == 0
