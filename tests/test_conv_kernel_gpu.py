"""DeltaNet layers with conv kernels other than four, against the CPU oracle: few rows of a short kernel leave the layer kernel
less to load than it has threads, a long one takes its general loop.  Bars as in test_spec_gpu.py."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
STEPS = 24


def _f(u):
    return np.array(u, dtype=np.uint32).view(np.float32)


@pytest.mark.parametrize("fast", [False, True], ids=["t-row", "dense-prompt"])
@pytest.mark.parametrize("k", [0, 1, 3])
@pytest.mark.parametrize("conv_kernel", [2, 3, 5, 8])
def test_conv_kernels(pkg, packs, oracle, llb, conv_kernel, k, fast):
    cfg = packs.cfg_tiny(conv_kernel=conv_kernel, seed=17)
    pack = packs.build_pack(cfg)
    prompt = packs.synth_prompt(2, 48 if fast else 10, cfg.vocab_size)   # ten tokens: chunks of eight rows and of one
    orc = oracle.Oracle(pack.index_text(), pack.data.numpy(), cap=len(prompt) + STEPS + 16)
    ref_ids, ref_top2 = orc.greedy(prompt, STEPS)
    mtp = packs.aux1_bytes(packs.build_mtp(pack)) if k else None
    eng = pkg.llb.SpecEngine(pack, mtp, k=k, max_ctx=len(prompt) + STEPS + 16)
    try:
        eng.set_prefill(fast)
        eng.prefill(prompt)
        assert (eng.fast_rows() > 0) == fast
        ids, top2 = eng.generate(STEPS)
    finally:
        eng.close()
    same = STEPS
    for i in range(STEPS):
        if ids[i] != ref_ids[i]:
            gap = float(_f(ref_top2[i][1]) - _f(ref_top2[i][3]))
            assert gap < 1e-3, f"token {i}: device {ids[i]}, oracle {ref_ids[i]}, oracle top-2 gap {gap}"
            same = i
            break
    v, r = _f(top2[:same, 1]), _f(ref_top2[:same, 1])
    assert np.all(np.abs(v - r) <= 2e-2 + 1e-2 * np.abs(r)), float(np.abs(v - r).max())
