"""The router's gate logits for many rows against those of the rows taken a few at a time: the same bits; and against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,E,d", [(2100, 128, 2048), (296 * 32, 4, 256), (259, 150, 512), (1185, 31, 768), (640, 512, 256)])
def test_logits_do_not_depend_on_the_number_of_rows(M, E, d):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from rexl3_b200.ops import lib
    L = lib.load()
    g = torch.Generator(device="cuda").manual_seed(M + E)
    x, gate = torch.randn(M, d, device="cuda", generator=g).bfloat16(), torch.randn(E, d, device="cuda", generator=g).bfloat16()

    def run(a, b):
        n = b - a
        lo, ids, w = torch.full((n + 1, E), -7.0, device="cuda"), torch.zeros(n, 1, dtype=torch.int32, device="cuda"), torch.zeros(n, 1, device="cuda")
        lib.check(L.rx_moe_router2(x[a:b].contiguous().data_ptr(), gate.data_ptr(), None, n, d, E, 1, 0, 1.0, lo.data_ptr(), ids.data_ptr(), w.data_ptr(),
                                   lib.stream_ptr()), "rx_moe_router2")
        assert (lo[n] == -7.0).all()
        return lo[:n], ids
    whole, ids = run(0, M)
    cut = [run(a, min(a + 31, M)) for a in range(0, M, 31)]
    assert torch.equal(whole, torch.cat([c[0] for c in cut])) and torch.equal(ids, torch.cat([c[1] for c in cut]))
    # one rounding (2^-24) per product-sum step of d terms at most
    bound = d * 2.0 ** -24 * (x.double().abs() @ gate.double().abs().T)
    assert ((whole.double() - x.double() @ gate.double().T).abs() <= bound).all()
