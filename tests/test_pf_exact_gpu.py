"""The dense GEMM on exact integer codes (k_pfx1 up to 128 prompt rows, k_pfx2 beyond for Q4_K and Q5_K) through llb_b200_pf_gemm, against
float64 dot products of the dequantised weights: row counts at the edges of its forms (units of 32, 64 and 128 rows), partial tiles of
weight rows, odd K-slices, and super-blocks whose scales differ by many orders of magnitude."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
# what two seeds show, 0.97 to 1.07, 1.07 to 1.22 and 1.26 to 1.36e-7, and 7 %: with 1 + 0.1 N the forty results of a weight row are nearly the same, so that the norm
# is that of 512 independent roundings, whose size goes with their mantissas (1.10 and 1.22e-7 for the two seeds)
BARS = (1.15e-7, 1.31e-7, 1.46e-7)


def _run(llb, packs, dev, ty, raw, rows, K, x, ksplit):
    L = llb.lib()
    fmt, R = packs.FMT[ty], x.shape[0]
    w = dev(L.llb_b200_weight_bytes(fmt, rows, K))
    llb.check(L.llb_b200_weight_upload(fmt, rows, K, raw.ctypes.data, 0, w.ptr), "weight_upload")
    xd, out = dev(x.nbytes).write(x), dev(R * rows * 4)
    llb.check(L.llb_b200_pf_gemm(fmt, w.ptr, rows, K, xd.ptr, R, out.ptr, ksplit), "llb_b200_pf_gemm")
    assert L.llb_b200_wait_errors() == 0
    return out.read((R, rows), np.float32).astype(np.float64)


@pytest.mark.parametrize("R", [1, 31, 32, 33, 64, 65, 128, 129, 255, 256])
@pytest.mark.parametrize("ty", ["Q4_K", "Q5_K", "Q6_K", "Q8_0"])
def test_edges_of_the_forms(llb, packs, oracle, dev, ty, R):
    rows, K, ksplit = 280 if R % 2 else 130, 1792 if R % 2 else 2048, 3 if R % 2 else 0   # slices of two and three super-blocks; a tile pair's second tile missing or partial
    rng = np.random.default_rng(R)
    raw = packs.QUANT[ty](torch.from_numpy(rng.standard_normal((rows, K), dtype=np.float32) * 0.05)).numpy()
    x = rng.standard_normal((R, K), dtype=np.float32)
    ref = x.astype(np.float64) @ oracle.Oracle.deq_rows(packs.FMT[ty], raw, rows, K).astype(np.float64).T
    got = _run(llb, packs, dev, ty, raw, rows, K, x, ksplit)
    # activations to 22 bits (2.4e-7 of a product at most); truncating chains of up to 33 additions (33 x 3e-8); Q6_K and Q8_0 beyond 128 rows are the
    # kernel of two rounded planes (chains of 3 x 128 additions: 1e-5)
    bar = 1e-5 if R > 128 and ty in ("Q6_K", "Q8_0") else 1.3e-6
    assert np.linalg.norm(got - ref) < bar * np.linalg.norm(ref)
    assert np.all(np.abs(got - ref) <= 1e-5 * (np.abs(x) @ np.abs(oracle.Oracle.deq_rows(packs.FMT[ty], raw, rows, K)).T) + 1e-6)


@pytest.mark.parametrize("R", [40, 200])
@pytest.mark.parametrize("ty", ["Q4_K", "Q5_K", "Q6_K", "Q8_0"])
def test_scales_of_many_magnitudes(llb, packs, oracle, dev, ty, R):
    """Blocks of 32 columns whose weights differ by up to six orders of magnitude; for Q4_K and Q5_K also blocks with d = 0, with no mins and with a dmin
    far above d, where the codes are taken a power of two smaller."""
    rows, K = 144, 1024
    rng = np.random.default_rng(5)
    mag = 10.0 ** rng.uniform(-4, 2, (rows, K // 32, 1)).astype(np.float32)
    raw = packs.QUANT[ty](torch.from_numpy((rng.standard_normal((rows, K // 32, 32), dtype=np.float32) * mag).reshape(rows, K))).numpy()
    fmt = packs.FMT[ty]
    mins = np.zeros((rows, K), np.float64)
    if ty in ("Q4_K", "Q5_K"):
        blk = raw.reshape(-1, 144 if ty == "Q4_K" else 176).copy()
        dd = blk[:, :4].copy().view(np.float16)
        dd[1::5, 0] = 0.0
        dd[2::5] = (1e-3, 6e4)
        dd[3::5, 1] = 0.0
        dd[4::5] = (6e-8, 1e-4)
        blk[:, :4] = dd.view(np.uint8)
        raw = blk.reshape(raw.shape)
        zero_d = blk.copy()
        zero_d[:, :2] = 0
        mins = np.abs(oracle.Oracle.deq_rows(fmt, zero_d.reshape(raw.shape), rows, K)).astype(np.float64)
    x = rng.standard_normal((R, K), dtype=np.float32)
    deq = oracle.Oracle.deq_rows(fmt, raw, rows, K).astype(np.float64)
    got = _run(llb, packs, dev, ty, raw, rows, K, x, 0)
    ref = x.astype(np.float64) @ deq.T
    # every product and every min term to about 1e-6 of itself (the kernel of two planes: 1e-5, and weights below 6e-5 to 6e-8 / 2048)
    mass = np.abs(x).astype(np.float64) @ (np.abs(deq) + 2 * mins).T
    bar = 1e-5 if R > 128 and ty in ("Q6_K", "Q8_0") else 3e-6
    assert np.all(np.abs(got - ref) <= bar * mass + 1e-6), float((np.abs(got - ref) / (mass + 1e-9)).max())


@pytest.mark.parametrize("power", [1, 3])
def test_sums_do_not_climb(llb, packs, oracle, dev, power):
    """Q6_K on activations of one sign, many columns: the planes of codes, of weights with heavy tails too, have no part that cancels between them and that truncated
    sums would add up."""
    rows, K = 512, 17408
    rng = np.random.default_rng(9)
    raw = packs.quant_q6_k(torch.from_numpy(rng.standard_normal((rows, K), dtype=np.float32) ** power * 0.02)).numpy()
    deq = oracle.Oracle.deq_rows(packs.FMT["Q6_K"], raw, rows, K).astype(np.float64)
    err = {}
    for kind in ("N", "|N|"):
        x = rng.standard_normal((40, K), dtype=np.float32)
        x = x if kind == "N" else np.abs(x)
        ref = x.astype(np.float64) @ deq.T
        err[kind] = np.linalg.norm(_run(llb, packs, dev, "Q6_K", raw, rows, K, x, 4) - ref) / np.linalg.norm(ref)
    assert err["|N|"] < 1.25 * err["N"], err


@pytest.mark.parametrize("ty", ["Q4_K", "Q5_K", "Q6_K", "Q8_0"])
def test_forms_give_the_same_bits(llb, packs, dev, ty):
    """A row's sums do not depend on how many rows come with it (up to 128: three forms of the kernel)."""
    rows, K = 400, 5120
    rng = np.random.default_rng(13)
    raw = packs.QUANT[ty](torch.from_numpy(rng.standard_normal((rows, K), dtype=np.float32) * 0.02)).numpy()
    x = rng.standard_normal((128, K), dtype=np.float32)
    got = [_run(llb, packs, dev, ty, raw, rows, K, x[:n], 3) for n in (20, 32, 33, 64, 65, 128)]
    for g in got[:-1]:
        assert np.array_equal(g, got[-1][:len(g)])


@pytest.mark.parametrize("ty", ["Q6_K", "Q8_0"])
@pytest.mark.parametrize("kind", ["N", "|N|", "silu", "1+.1N"])
def test_error_against_64_bits(llb, packs, oracle, dev, ty, kind):
    """The formats whose T-row passes are exact but for the activations' 22 bits and fp32 sums (1.0e-7 to 1.2e-7 of Q6_K, 0.9e-7 to 2.0e-7 of Q8_0), at the K-slices that
    a prompt takes."""
    rng = np.random.default_rng(17)
    for rows, K, ksplit, bar in ((512, 1024, 4, BARS[0]), (512, 5120, 3, BARS[1]), (512, 17408, 3, BARS[2])):
        raw = packs.QUANT[ty](torch.from_numpy(rng.standard_normal((rows, K), dtype=np.float32) * 0.02)).numpy()
        r = rng.standard_normal((40, K), dtype=np.float32)
        x = {"N": r, "|N|": np.abs(r), "1+.1N": 1 + np.float32(0.1) * r, "silu": r / (1 + np.exp(-r)) * rng.standard_normal((40, K), dtype=np.float32)}[kind]
        ref = x.astype(np.float64) @ oracle.Oracle.deq_rows(packs.FMT[ty], raw, rows, K).astype(np.float64).T
        err = np.linalg.norm(_run(llb, packs, dev, ty, raw, rows, K, x, ksplit) - ref) / np.linalg.norm(ref)
        assert err < bar, (K, err)
