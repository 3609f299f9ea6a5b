"""Programmatic launches must not show in the results: with them on, a kernel's blocks are resident long before their
producer runs, and a plain load of a buffer that every layer rewrites may meet an earlier layer's line in the SM's L1.  Each
run is a process of its own (the switch is read when the library is initialised); the bits of both must be the same."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

RUN = """
import hashlib, sys
import numpy as np
import __graft_entry__ as graft
pkg = graft.load_package()
llb, packs = pkg.llb, pkg.packs
llb.init(0)
what = sys.argv[1]
h = hashlib.sha256()
def add(*arrays):
    for a in arrays:
        h.update(np.ascontiguousarray(a).tobytes())
if what == "experts" or what == "expert-streams":
    cfg = packs.cfg_tiny_moe(n_layers=24, mix_gain=0.1)
    mtp = None
else:
    cfg = packs.cfg_tiny(n_layers=24, mix_gain=0.1, vocab_size=2048)
pack = packs.build_pack(cfg)
if cfg.n_experts == 0:
    mtp = packs.aux1_bytes(packs.build_mtp(pack))
if what == "expert-streams":
    eng = llb.SpecEngine(pack, None, k=1, max_ctx=128, streams=8)
    for b in range(8):
        eng.prefill_stream(b, packs.synth_prompt(b, 9 + 3 * b, cfg.vocab_size))
    for _ in range(12):
        for i, t in eng.cycle_streams():
            add(i, t)
else:
    eng = llb.SpecEngine(pack, mtp, k=3, max_ctx=256)
    if what == "sampled":
        eng.set_sampler(llb.SmpParams.make(temp=0.8, top_p=0.95, top_k=40, repeat_penalty=1.1, seed=5))
    eng.prefill(packs.synth_prompt(7, 61, cfg.vocab_size))
    add(*eng.generate(64))
print("bits", h.hexdigest())
"""


@pytest.mark.parametrize("what", ["experts", "expert-streams", "drafter", "sampled"])
def test_results_do_not_depend_on_programmatic_launches(what):
    bits = []
    for pdl in ("0", "1", "1"):
        r = subprocess.run([sys.executable, "-c", RUN, what], cwd=ROOT, env=dict(os.environ, LLB_PDL=pdl, PYTHONPATH=ROOT), capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr[-2000:]
        bits.append([l for l in r.stdout.splitlines() if l.startswith("bits")][0])
    assert bits[0] == bits[1] == bits[2]
