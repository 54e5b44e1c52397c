"""The tensor-core GEMM that reads weight planes (tc_kernel): edges of its tiles (128 features, 16 to 256 tokens), of its plane
chunks (512 or 256 features), K runs split over CTAs and whole tiles, every weight width.  int32 results bit for bit against the
oracle's exact product; the fp16 epilogues against float64 (check_close's bound: the fp16 rounding of the result, and with
per-group scales the fp32 sums over the groups)."""
import numpy as np
import pytest

from helpers import dev, planes_dev, rand_codes, run_gemm
from test_gpu_gemm_fp16 import check_close

pytestmark = pytest.mark.gpu

INT_CASES = [
    # M, N, K, x_bits, w_bits, x_signed, w_signed
    (1, 128, 128, 8, 1, True, False), (16, 130, 640, 4, 2, True, True), (17, 127, 1152, 8, 3, True, True), (32, 1000, 512, 3, 4, False, False),
    (33, 4096, 4096, 4, 4, False, False), (64, 257, 2944, 6, 5, True, True), (65, 4100, 1408, 6, 6, True, False), (128, 384, 256, 7, 7, True, True),
    (129, 1001, 896, 8, 8, True, True), (256, 4096, 384, 8, 8, False, False), (257, 300, 4096, 2, 8, True, False), (1024, 129, 2048, 5, 1, True, True),
]


@pytest.mark.parametrize("split", [0, 1])
@pytest.mark.parametrize("case", INT_CASES, ids=lambda c: "M{}N{}K{}a{}w{}{}{}".format(*c[:5], "s" if c[5] else "u", "s" if c[6] else "u"))
def test_int32(abq, oracle, cuda, case, split, monkeypatch):
    monkeypatch.setenv("ABQ_TC_SPLIT", str(split))
    M, N, K, p, q, xs, ws = case
    rng = np.random.default_rng(M + N + K + q)
    x, w = rand_codes(rng, M, K, p, xs), rand_codes(rng, N, K, q, ws)
    got, st = run_gemm(abq, planes_dev(oracle, x, p), planes_dev(oracle, w, q), M, N, K, x_bits=p, w_bits=q, x_signed=xs, w_signed=ws,
                       route=abq.ROUTE_I8_UMMA)
    want = oracle.gemm_values_blas(x, w)
    assert np.array_equal(got, want), f"{np.count_nonzero(got != want)} of {got.size} differ"


@pytest.mark.parametrize("bt", [16, 32, 64, 128])
@pytest.mark.parametrize("M,N,K,q,group,xs,with_zero", [(16, 200, 1024, 2, 64, True, True), (61, 520, 2944, 4, 128, True, True),
                                                        (130, 300, 1280, 3, 640, True, True), (40, 256, 1536, 8, 64, False, False),
                                                        (100, 129, 640, 7, 128, False, True)])
def test_scale_groups(abq, oracle, cuda, M, N, K, q, group, xs, with_zero, bt, monkeypatch):
    """Odd group counts, groups of half a K block and of several, unsigned x unsigned sums above 2^22, K runs cut inside a group."""
    monkeypatch.setenv("ABQ_TC_BT", str(bt))
    rng = np.random.default_rng(M + K + q)
    x, w = rand_codes(rng, M, K, 8, xs), rand_codes(rng, N, K, q, False)
    G = K // group
    scale = rng.uniform(0.001, 0.02, size=(N, G)).astype(np.float16)
    zero = rng.integers(0, 1 << q, size=(N, G)).astype(np.uint8) if with_zero else None
    tok = rng.uniform(0.001, 0.01, size=M).astype(np.float32)
    for split in ("0", "1"):
        monkeypatch.setenv("ABQ_TC_SPLIT", split)
        got, st = run_gemm(abq, planes_dev(oracle, x, 8), planes_dev(oracle, w, q), M, N, K, x_bits=8, w_bits=q, x_signed=xs, w_signed=False,
                           out_fp16=True, scale_mode=abq.SCALE_GROUP, group_size=group, w_scale=dev(scale),
                           w_zero=None if zero is None else dev(zero), x_scale=dev(tok), route=abq.ROUTE_I8_UMMA)
        check_close(got, oracle.dequant_gemm(x, w, scale, None if zero is None else zero.astype(np.int32), tok, group))


@pytest.mark.parametrize("q,w_signed", [(1, False), (2, True), (3, False), (3, True), (4, False), (5, True), (7, False), (8, False), (8, True)])
def test_channel_zero_points(abq, oracle, cuda, q, w_signed):
    """Zero points subtracted in the codes (up to three bits, unsigned) or times the token's code sum, K runs cut or not; two tiles of
    tokens, the second one ragged."""
    M, N, K = 70, 300, 1408
    rng = np.random.default_rng(q)
    x, w = rand_codes(rng, M, K, 8, True), rand_codes(rng, N, K, q, w_signed)
    scale = rng.uniform(0.001, 0.02, size=N).astype(np.float16)
    zero = rng.integers(0, 1 << q, size=N, dtype=np.uint8)
    xs = rng.uniform(0.05, 0.2, size=M).astype(np.float32)
    got, st = run_gemm(abq, planes_dev(oracle, x, 8), planes_dev(oracle, w, q), M, N, K, x_bits=8, w_bits=q, x_signed=True, w_signed=w_signed,
                       route=abq.ROUTE_I8_UMMA, out_fp16=True, scale_mode=abq.SCALE_CHANNEL, w_scale=dev(scale), w_zero=dev(zero), x_scale=dev(xs))
    acc = oracle.gemm_values_blas(x, w).astype(np.float64) - zero.astype(np.float64)[None, :] * x.sum(axis=1, dtype=np.int64)[:, None]
    check_close(got, acc * scale.astype(np.float64)[None, :] * xs.astype(np.float64)[:, None])


@pytest.mark.parametrize("M", [24, 100, 200])
def test_scales_of_groups_of_64_off_a_word(abq, oracle, cuda, M):
    """fp16 scales that start two bytes off a 32-bit word (a view into a larger buffer) give the bits that an aligned copy gives,
    over planes (24, 100 rows) and over expanded codes (200)."""
    N, K, q, group = 200, 1152, 3, 64
    rng = np.random.default_rng(M)
    x, w = rand_codes(rng, M, K, 8, True), rand_codes(rng, N, K, q, False)
    G = K // group
    flat = dev(rng.uniform(0.001, 0.02, size=N * G + 2).astype(np.float16))
    off = flat[1:1 + N * G].view(N, G)
    assert off.data_ptr() % 4 == 2 and off.is_contiguous()
    aligned = off.clone()
    zero = rng.integers(0, 1 << q, size=(N, G)).astype(np.uint8)
    tok = rng.uniform(0.001, 0.01, size=M).astype(np.float32)
    got = []
    for scale in (aligned, off):
        d, st = run_gemm(abq, planes_dev(oracle, x, 8), planes_dev(oracle, w, q), M, N, K, x_bits=8, w_bits=q, x_signed=True, w_signed=False,
                         out_fp16=True, scale_mode=abq.SCALE_GROUP, group_size=group, w_scale=scale, w_zero=dev(zero), x_scale=dev(tok),
                         route=abq.ROUTE_I8_UMMA)
        got.append(d)
    check_close(got[0], oracle.dequant_gemm(x, w, aligned.cpu().numpy(), zero.astype(np.int32), tok, group))
    assert np.array_equal(got[0].view(np.uint16), got[1].view(np.uint16))


@pytest.mark.parametrize("M,N,group,want", [(32, 4096, 0, "tc_kernel"), (200, 256, 0, "tc_kernel"), (512, 256, 0, "umma_kernel"), (512, 257, 0, "tc_kernel"),
                                            (100, 256, 64, "tc_kernel"), (200, 256, 128, "tc_kernel (codes)")])
def test_the_kernel_a_plan_reports(abq, oracle, cuda, M, N, group, want):
    K = 4096
    rng = np.random.default_rng(N)
    kw = dict(out_fp16=True, scale_mode=abq.SCALE_GROUP, group_size=group, w_scale=dev(np.ones((N, K // group), dtype=np.float16))) if group else {}
    _, st = run_gemm(abq, planes_dev(oracle, rand_codes(rng, M, K, 2, True), 2), planes_dev(oracle, rand_codes(rng, N, K, 2, False), 2), M, N, K,
                     x_bits=2, w_bits=2, x_signed=True, w_signed=False, **kw)
    assert abq.state_kernel(st) == want


@pytest.mark.parametrize("split", [0, 1])
@pytest.mark.parametrize("M,N,K,group", [(16, 1024, 4096, 256), (16, 1024, 4096, 1024), (16, 2048, 3840, 640), (100, 300, 3072, 3072), (200, 300, 1536, 512),
                                         (16, 1024, 4096, 4096)])
def test_wide_groups_are_summed_whole(abq, oracle, cuda, M, N, K, group, split, monkeypatch):
    """Groups of more than 128 features are summed as whole numbers and rounded once, however K is cut.  Here the two halves of a group
    almost cancel: the sum is 1 to 3, the halves reach 3.9e6 x group / 256, of which a product with the scale that is rounded to fp32 per 128
    features keeps 24 bits, i.e. an error of a tenth of the result and more.  The exact sums leave the fp32 rounding of the sum over
    groups (relative 2^-24 each, all terms positive) and of the result (2^-11)."""
    monkeypatch.setenv("ABQ_TC_SPLIT", str(split))
    rng = np.random.default_rng(group + M)
    half, G = group // 2, K // group
    x = np.empty((M, G, 2, half), dtype=np.int32)
    w = np.empty((N, G, 2, half), dtype=np.int32)
    x[:, :, 0] = rng.integers(120, 128, size=(M, G, half))
    w[:, :, 0] = rng.integers(200, 256, size=(N, G, half))
    x[:, :, 0, 0] = rng.integers(1, 4, size=(M, G))
    x[:, :, 1], w[:, :, 1] = -x[:, :, 0], w[:, :, 0]
    w[:, :, 1, 0] -= 1
    x, w = x.reshape(M, K), w.reshape(N, K)
    scale = rng.uniform(0.001, 0.02, size=(N, G)).astype(np.float16)
    got, st = run_gemm(abq, planes_dev(oracle, x, 8), planes_dev(oracle, w, 8), M, N, K, x_bits=8, w_bits=8, x_signed=True, w_signed=False,
                       out_fp16=True, scale_mode=abq.SCALE_GROUP, group_size=group, w_scale=dev(scale), route=abq.ROUTE_I8_UMMA)
    assert abq.state_kernel(st) == ("tc_kernel" if M <= 128 else "tc_kernel (codes)")
    ref = oracle.dequant_gemm(x, w, scale, None, np.ones(M, dtype=np.float32), group)
    assert np.all(np.abs(got.astype(np.float64) - ref) <= (2.0 ** -11 + 2.0 ** -24 * (G + 2)) * np.abs(ref))
