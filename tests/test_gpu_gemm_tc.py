"""The tensor-core GEMM that reads weight planes (tc_kernel): edges of its tiles (128 features, 16 to 256 tokens), of its plane
chunks (512 or 256 features), K runs split over CTAs and whole tiles, every weight width.  int32 results bit for bit against the
oracle's exact product; the fp16 epilogues against float64 (check_close's bound: the fp16 rounding of the result, and with
per-group scales the fp32 sums over the groups)."""
import numpy as np
import pytest

from helpers import dev, planes_dev, rand_codes, run_gemm
from test_gpu_gemm_fp16 import check_close

pytestmark = pytest.mark.gpu

def plan_of(abq, st):
    """(kernel, tokens per tile, K cut over CTAs) of a plan."""
    return abq.state_kernel(st), st.tile[3], bool(st.tile[1])


def force(monkeypatch, bt, split):
    monkeypatch.setenv("ABQ_TC_BT", str(bt))
    monkeypatch.setenv("ABQ_TC_SPLIT", str(int(split)))


INT_CASES = [
    # tokens per tile, K cut, M, N, K, x_bits, w_bits, x_signed, w_signed
    (32, False, 1, 128, 128, 8, 1, True, False), (32, False, 16, 130, 640, 4, 2, True, True), (64, False, 17, 127, 1152, 8, 3, True, True),
    (256, False, 32, 1000, 512, 3, 4, False, False), (32, False, 33, 4096, 4096, 4, 4, False, False), (128, False, 64, 257, 2944, 6, 5, True, True),
    (64, False, 65, 4100, 1408, 6, 6, True, False), (128, False, 128, 384, 256, 7, 7, True, True), (256, False, 129, 1001, 896, 8, 8, True, True),
    (256, False, 256, 4096, 384, 8, 8, False, False), (256, False, 257, 301, 4096, 2, 8, True, False), (256, False, 1024, 129, 2048, 5, 1, True, True),
    # cut tiles: sizes whose partial tiles fit into the scratch
    (32, True, 1, 384, 2048, 8, 1, True, False), (32, True, 17, 257, 1408, 4, 2, True, True), (32, True, 33, 1000, 8192, 8, 3, True, True),
    (128, True, 65, 4100, 8192, 4, 4, False, False), (64, True, 64, 4097, 4096, 6, 5, True, True), (256, True, 200, 4865, 8192, 6, 6, True, True),
    (128, True, 129, 2561, 8192, 7, 7, True, False), (32, True, 20, 1001, 8192, 8, 8, False, False), (256, True, 200, 4865, 8192, 4, 4, True, True),
]


@pytest.mark.parametrize("case", INT_CASES, ids=lambda c: "bt{}{}-M{}N{}K{}a{}w{}{}{}".format(c[0], "cut" if c[1] else "", *c[2:7], "s" if c[7] else "u",
                                                                                           "s" if c[8] else "u"))
def test_int32(abq, oracle, cuda, case, monkeypatch):
    bt, split, M, N, K, p, q, xs, ws = case
    force(monkeypatch, bt, split)
    rng = np.random.default_rng(M + N + K + q)
    x, w = rand_codes(rng, M, K, p, xs), rand_codes(rng, N, K, q, ws)
    got, st = run_gemm(abq, planes_dev(oracle, x, p), planes_dev(oracle, w, q), M, N, K, x_bits=p, w_bits=q, x_signed=xs, w_signed=ws,
                       route=abq.ROUTE_I8_UMMA)
    assert plan_of(abq, st) == ("tc_kernel", bt, split)
    want = oracle.gemm_values_blas(x, w)
    assert np.array_equal(got, want), f"{np.count_nonzero(got != want)} of {got.size} differ"


@pytest.mark.parametrize("M,N,K", [(1, 2048, 4096), (100, 10007, 2944), (256, 4096, 1024), (300, 1001, 2048)])
def test_int32_as_planned(abq, oracle, cuda, M, N, K):
    """The planner's own choice of tile and cut."""
    rng = np.random.default_rng(M)
    x, w = rand_codes(rng, M, K, 4, True), rand_codes(rng, N, K, 4, False)
    got, st = run_gemm(abq, planes_dev(oracle, x, 4), planes_dev(oracle, w, 4), M, N, K, x_bits=4, w_bits=4, x_signed=True, w_signed=False,
                       route=abq.ROUTE_I8_UMMA)
    assert plan_of(abq, st)[0] == "tc_kernel"
    assert np.array_equal(got, oracle.gemm_values_blas(x, w))


@pytest.mark.parametrize("bt", [16, 32, 64])
@pytest.mark.parametrize("M,N,K,q,group,xs,with_zero", [(16, 1300, 8192, 2, 64, True, True), (61, 1300, 8192, 4, 128, True, True),
                                                        (100, 1300, 5120, 3, 640, True, True), (40, 1300, 8192, 8, 64, False, False),
                                                        (100, 1300, 8192, 7, 128, False, True), (33, 1301, 8320, 5, 64, True, True)])
def test_scale_groups(abq, oracle, cuda, M, N, K, q, group, xs, with_zero, bt, monkeypatch):
    """Odd group counts, groups of half a K block and of several, unsigned x unsigned sums above 2^22, K cut or not, inside runs of groups."""
    rng = np.random.default_rng(M + K + q)
    x, w = rand_codes(rng, M, K, 8, xs), rand_codes(rng, N, K, q, False)
    G = K // group
    scale = rng.uniform(0.001, 0.02, size=(N, G)).astype(np.float16)
    zero = rng.integers(0, 1 << q, size=(N, G)).astype(np.uint8) if with_zero else None
    tok = rng.uniform(0.001, 0.01, size=M).astype(np.float32)
    ref = oracle.dequant_gemm(x, w, scale, None if zero is None else zero.astype(np.int32), tok, group)
    xp, wp = planes_dev(oracle, x, 8), planes_dev(oracle, w, q)
    for split in (False, True):
        force(monkeypatch, bt, split)
        got, st = run_gemm(abq, xp, wp, M, N, K, x_bits=8, w_bits=q, x_signed=xs, w_signed=False, out_fp16=True, scale_mode=abq.SCALE_GROUP,
                           group_size=group, w_scale=dev(scale), w_zero=None if zero is None else dev(zero), x_scale=dev(tok), route=abq.ROUTE_I8_UMMA)
        assert plan_of(abq, st) == ("tc_kernel", bt, split)
        check_close(got, ref)


@pytest.mark.parametrize("M,K,q,group", [(130, 1280, 3, 640), (129, 1152, 4, 64), (300, 1408, 7, 128)])
def test_scale_groups_over_expanded_codes(abq, oracle, cuda, M, K, q, group):
    N = 300
    rng = np.random.default_rng(M + K + q)
    x, w = rand_codes(rng, M, K, 8, True), rand_codes(rng, N, K, q, False)
    scale = rng.uniform(0.001, 0.02, size=(N, K // group)).astype(np.float16)
    zero = rng.integers(0, 1 << q, size=(N, K // group)).astype(np.uint8)
    tok = rng.uniform(0.001, 0.01, size=M).astype(np.float32)
    got, st = run_gemm(abq, planes_dev(oracle, x, 8), planes_dev(oracle, w, q), M, N, K, x_bits=8, w_bits=q, x_signed=True, w_signed=False,
                       out_fp16=True, scale_mode=abq.SCALE_GROUP, group_size=group, w_scale=dev(scale), w_zero=dev(zero), x_scale=dev(tok))
    assert plan_of(abq, st) == ("tc_kernel (codes)", 128, False)
    check_close(got, oracle.dequant_gemm(x, w, scale, zero.astype(np.int32), tok, group))


@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("q,w_signed", [(1, False), (2, True), (3, False), (3, True), (4, False), (5, True), (7, False), (8, False), (8, True)])
def test_channel_zero_points(abq, oracle, cuda, q, w_signed, split, monkeypatch):
    """Zero points subtracted in the codes (two and three bits, unsigned) or times the token's code sum, K cut or not; tiles of 32
    tokens, the last one ragged."""
    M, N, K = 70, 700, 8192
    force(monkeypatch, 32, split)
    rng = np.random.default_rng(q)
    x, w = rand_codes(rng, M, K, 8, True), rand_codes(rng, N, K, q, w_signed)
    scale = rng.uniform(0.001, 0.02, size=N).astype(np.float16)
    zero = rng.integers(0, 1 << q, size=N, dtype=np.uint8)
    xs = rng.uniform(0.05, 0.2, size=M).astype(np.float32)
    got, st = run_gemm(abq, planes_dev(oracle, x, 8), planes_dev(oracle, w, q), M, N, K, x_bits=8, w_bits=q, x_signed=True, w_signed=w_signed,
                       route=abq.ROUTE_I8_UMMA, out_fp16=True, scale_mode=abq.SCALE_CHANNEL, w_scale=dev(scale), w_zero=dev(zero), x_scale=dev(xs))
    assert plan_of(abq, st) == ("tc_kernel", 32, split)
    acc = oracle.gemm_values_blas(x, w).astype(np.float64) - zero.astype(np.float64)[None, :] * x.sum(axis=1, dtype=np.int64)[:, None]
    check_close(got, acc * scale.astype(np.float64)[None, :] * xs.astype(np.float64)[:, None])


@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("M,q", [(17, 4), (25, 2), (32, 8)])
@pytest.mark.parametrize("mode", ["channel", "tensor"])
def test_residual_by_auto(abq, oracle, cuda, M, q, mode, split, monkeypatch):
    """AUTO at 17 to 32 rows plans tc_kernel for large matrices, with its residual input: the fp16 add of the result without one."""
    from abq_llm_b200 import binding as B
    N, K = 4096, 4096
    force(monkeypatch, 32, split)
    rng = np.random.default_rng(M)
    x, w = rand_codes(rng, M, K, 8, True), rand_codes(rng, N, K, q, False)
    if mode == "tensor":
        x = np.fix(x / 64).astype(np.int32)  # sums that fp16 holds
    kw = dict(scale_mode=abq.SCALE_TENSOR_COMPAT, C=dev(np.array([0.0023], dtype=np.float16)))
    if mode == "channel":
        kw = dict(scale_mode=abq.SCALE_CHANNEL, w_scale=dev(rng.uniform(1e-4, 1e-3, size=N).astype(np.float16)),
                  w_zero=dev(rng.integers(0, 1 << q, size=N, dtype=np.uint8)), x_scale=dev(rng.uniform(0.05, 0.2, size=M).astype(np.float32)))
    ws = dev(np.zeros(abq.gemm_workspace_bytes(M, N, K, 8, q), dtype=np.uint8))
    xp, wp = planes_dev(oracle, x, 8), planes_dev(oracle, w, q)
    res = rng.normal(0, 1, size=(M, N)).astype(np.float16)
    outs = []
    for residual in (None, dev(res)):
        out = dev(np.zeros((M, N), dtype=np.float16))
        prm = B.make_params(M, N, K, xp, wp, out, x_bits=8, w_bits=q, x_signed=True, w_signed=False, out_dtype=abq.OUT_FP16, workspace=ws,
                            residual=residual, **kw)
        st = abq.gemm_init(prm)
        assert plan_of(abq, st) == ("tc_kernel", 32, split)
        abq.gemm_exec(st)
        outs.append(out.cpu().numpy())
    assert np.isfinite(outs[0].astype(np.float32)).all() and np.abs(outs[0]).max() > 0.1
    assert np.array_equal(outs[1].view(np.uint16), (outs[0] + res).view(np.uint16))


@pytest.mark.parametrize("q", [2, 3, 4])
@pytest.mark.parametrize("M", [20, 100])
def test_fp16_activations(abq, oracle, cuda, M, q):
    """ABQ_FLAG_X_HALF: the codes written in the order of the weights' expansion (its own for two and three bits) give the bits that
    the quantiser's planes give, and the oracle's result."""
    from abq_llm_b200 import binding as B
    N, K, p = 1000, 1152, 8
    rng = np.random.default_rng(M + q)
    x = dev(rng.normal(0, 1, size=(M, K)).astype(np.float16))
    w = rand_codes(rng, N, K, q, False)
    qs = dev(np.array([20.0], dtype=np.float32))
    planes = dev(np.zeros((p, M, K // 32), dtype=np.int32))
    abq.quantize_pack_half(x, qs, planes, M, K, p, 0)
    wp, ws = planes_dev(oracle, w, q), dev(np.zeros(abq.gemm_workspace_bytes(M, N, K, p, q, abq.ROUTE_I8_UMMA), dtype=np.uint8))
    outs = []
    for X, flags in ((planes, 0), (x, abq.FLAG_X_HALF)):
        out = dev(np.zeros((M, N), dtype=np.int32))
        prm = B.make_params(M, N, K, X, wp, out, x_bits=p, w_bits=q, x_signed=True, w_signed=False, route=abq.ROUTE_I8_UMMA, flags=flags,
                            x_quant_scale=qs, workspace=ws)
        st = abq.gemm_init(prm)
        assert plan_of(abq, st)[0] == "tc_kernel"
        abq.gemm_exec(st)
        outs.append(out.cpu().numpy())
    assert np.array_equal(outs[0], oracle.gemm_values_blas(oracle.unpack(planes.cpu().numpy().view(np.uint32), True), w))
    assert np.array_equal(outs[0], outs[1])


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
