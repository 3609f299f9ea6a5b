"""The prompt path's attention (k_pf_attn) against the T-row passes' (k_attn_mma) on the same model: both head dimensions, one to eight query
heads a kv head, row counts that end inside, at and just past a block of 128 queries and a tile of 32 positions, pieces behind earlier
ones, and a context long enough for many slices of a piece of few rows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FORMS = [dict(n_heads=2, n_kv_heads=2, head_dim=128), dict(n_heads=6, n_kv_heads=1, head_dim=256), dict(n_heads=8, n_kv_heads=1, head_dim=128)]
LENS = [16, 21, 22, 32, 33, 63, 128, 161, 290]


def _run(pkg, pack, prompt, mode):
    cfg = pack.cfg
    eng = pkg.llb.SpecEngine(pack, None, k=0, max_ctx=len(prompt) + 32)
    try:
        eng.set_prefill(mode)
        eng.prefill(prompt)
        n = len(prompt)
        st = {f"kv{what}.{il}": np.stack([eng.read_state(what, il, p) for p in range(0, n - 1, 1 + n // 40)]) for il in range(cfg.n_layers) if cfg.is_full(il) for what in (1, 2)}
        st["lg"] = eng.read_logits(0)
        assert pkg.llb.lib().llb_b200_wait_errors() == 0
        return st
    finally:
        eng.close()


def _check(pkg, pack, monkeypatch, prompt):
    got = {m: _run(pkg, pack, prompt, m) for m in (False, True)}
    monkeypatch.setenv("LLB_PREFILL_ROWS", "8")
    ref = _run(pkg, pack, prompt, False)
    # the full layers' K and V carry the attention of those before; a query has 22 bits in both kernels, what differs is the order of the sums (the
    # dense GEMMs' too, 1e-5 of a row at most where mode 1 takes the kernel of rounded planes), amplified by the layers
    for m in got:
        for key, v in ref.items():
            d = np.abs(got[m][key] - v)
            assert np.all(d <= 2e-4 + 1e-3 * np.abs(v)), (m, key, float(d.max()))


@pytest.mark.parametrize("n", LENS)
@pytest.mark.parametrize("form", range(len(FORMS)))
def test_rows_and_tiles(pkg, packs, llb, monkeypatch, form, n):
    pack = packs.build_pack(packs.cfg_tiny(n_layers=8, seed=41 + form, **FORMS[form]))
    _check(pkg, pack, monkeypatch, packs.synth_prompt(n, n, pack.cfg.vocab_size))


def test_many_slices(pkg, packs, llb, monkeypatch):
    """A last piece of ten rows behind 12800 positions: 37 slices, more than the lanes that hold their weights."""
    pack = packs.build_pack(packs.cfg_tiny(n_layers=4, seed=51, **FORMS[1]))
    _check(pkg, pack, monkeypatch, packs.synth_prompt(3, 12800 + 11, pack.cfg.vocab_size))
