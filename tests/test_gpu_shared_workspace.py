"""Plans that share one workspace, called in turn.  A decode plan that splits K keeps its arrival counters in the workspace, cleared
once when the plan is made; no launch of another plan may leave something else there, whatever its route or its size.  A call whose
counters are not zero leaves its output as it was, so every call gets new activations and is compared whole."""
import numpy as np
import pytest
import torch

from helpers import dev, planes_dev, rand_codes

pytestmark = pytest.mark.gpu


class Plan:
    def __init__(self, abq, oracle, rng, M, N, K, bits, ws, codes, planes, flags=0, route=0, **kw):
        from abq_llm_b200 import binding as B
        self.abq, self.oracle, self.rng, self.M, self.K, self.bits, self.codes = abq, oracle, rng, M, K, bits, codes
        self.X = torch.empty((bits, M, K // 32), dtype=torch.int32, device="cuda")
        self.out = torch.full((M, N), -7, dtype=torch.int32, device="cuda")
        self.status = torch.zeros(1, dtype=torch.int32, device="cuda")
        self.params = B.make_params(M, N, K, self.X, planes, self.out, x_bits=bits, w_bits=bits, x_signed=True, w_signed=False,
                                    workspace=ws, status_word=self.status, flags=flags, route=route, **kw)  # (keeps its tensors)
        self.state = abq.gemm_init(self.params)

    def check(self):
        x = rand_codes(self.rng, self.M, self.K, self.bits, True)
        self.X.copy_(planes_dev(self.oracle, x, self.bits))
        self.abq.gemm_exec(self.state)
        torch.cuda.synchronize()
        assert int(self.status.item()) == 0
        assert np.array_equal(self.out.cpu().numpy(), self.oracle.gemm_values_blas(x, self.codes)), f"{self.M} rows"


@pytest.mark.parametrize("rows", [(16, 32, 64, 300), (16, 32, 128)])
def test_row_counts_in_turn(abq, oracle, cuda, rows):
    """Split K (16 rows), the tensor-core kernel over planes (32 rows by AUTO's rule for 16 Mi weights and more; 64) and over expanded codes
    (300) on one workspace, which the largest asks for.  Up to 128 rows that has no room of its own for the counters."""
    N, K, bits = 1536, 11008, 4
    rng = np.random.default_rng(7)
    w = rand_codes(rng, N, K, bits, False)
    planes = planes_dev(oracle, w, bits)
    ws = torch.full((abq.gemm_workspace_bytes(rows[-1], N, K, bits, bits),), 0xA5, dtype=torch.uint8, device="cuda")
    plans = {M: Plan(abq, oracle, rng, M, N, K, bits, ws, w, planes) for M in rows}
    assert plans[16].state.route == abq.ROUTE_I8_MMA and plans[16].state.cluster > 1, "meant to split K"
    assert plans[32].state.route == abq.ROUTE_I8_UMMA
    for M in [r for m in rows[1:] for r in (16, m)] + [16]:
        plans[M].check()


@pytest.mark.parametrize("small", [3072, 4000])
def test_matrices_of_different_sizes_at_decode_sizes(abq, oracle, cuda, small):
    """Two split plans in the workspace that the larger one asks for: the smaller one's partial tiles lie behind the larger one's counters."""
    K, bits = 11008, 4
    rng = np.random.default_rng(small)
    ws = torch.full((abq.gemm_workspace_bytes(5, 4096, K, bits, bits),), 0xA5, dtype=torch.uint8, device="cuda")
    plans = []
    for N in (4096, small):
        w = rand_codes(rng, N, K, bits, False)
        plans.append(Plan(abq, oracle, rng, 5, N, K, bits, ws, w, planes_dev(oracle, w, bits)))
    assert all(p.state.cluster > 1 for p in plans), "meant to split K"
    for i in (0, 1, 0, 1):
        plans[i].check()


def test_matrices_of_different_sizes(abq, oracle, cuda):
    """The counters of the larger matrix reach further than those of the smaller one."""
    K, bits = 11008, 4
    rng = np.random.default_rng(8)
    ws = torch.full((max(abq.gemm_workspace_bytes(M, N, K, bits, bits) for M, N in ((16, 4096), (64, 256))),), 0xA5, dtype=torch.uint8, device="cuda")
    plans = []
    for N in (4096, 256):
        w = rand_codes(rng, N, K, bits, False)
        planes = planes_dev(oracle, w, bits)
        plans += [Plan(abq, oracle, rng, M, N, K, bits, ws, w, planes) for M in ((16,) if N == 4096 else (16, 64))]
    assert plans[0].state.cluster > 1 and plans[1].state.cluster > 1, "meant to split K"
    for i in (0, 1, 0, 2, 0, 1):
        plans[i].check()


@pytest.mark.parametrize("group", [0, 128])
def test_linear_layer_with_changing_row_counts(abq, cuda, group):
    """A layer of the block linears keeps one workspace for all of its token counts: each call gives what a layer of its own gives."""
    from test_tp_linear_gloo import _tp
    tp = _tp()
    N, K, bits = 4096, 11008, 4
    g = torch.Generator(device="cuda")
    g.manual_seed(9)
    codes = torch.randint(0, 16, (N, K), dtype=torch.int32, device="cuda", generator=g)
    shape = (N, K // group) if group else (N,)
    scale = (torch.rand(shape, device="cuda", generator=g) * 0.01 + 0.001).half()
    zero = torch.randint(7, 10, shape, dtype=torch.int32, device="cuda", generator=g).to(torch.uint8)
    backend = tp.AbqBackend(abq, torch, None, x_bits=4, x_scale=2.0, max_tokens=300)
    shared = backend.make_linear(codes, scale, zero, bits, group)
    own = {}
    for i, M in enumerate((16, 32, 16, 64, 16, 300, 16, 20, 9, 300)):
        if M not in own:
            own[M] = backend.make_linear(codes, scale, zero, bits, group)
        x = torch.randn((M, K), device="cuda", generator=g).half()
        want = own[M](x).clone()
        assert torch.equal(shared(x), want), f"call {i}, {M} rows"
    torch.cuda.synchronize()
    assert int(backend.status.item()) == 0
