"""Simple lattices and their gradients on confident logits: where the am row and the lm row peak at
different symbols the normalizer is small because its terms are, far below what fp16 planes of
exp(x - max) hold.  Against the float64 path, for vocabularies of every kind.

Lattices: 1e-5, and 1e-6 of the entry for the roundings of a few float32 values of its size.
Gradients: 2e-5 of the norm."""
import pytest
import torch

from tests.test_odd_vocabulary_gpu import lattices

pytestmark = pytest.mark.gpu


def check(lm, am, symbols, rnnt_type, scales, seed, dtype=torch.float32):
    got = lattices(lm.to(dtype), am.to(dtype), symbols, rnnt_type, scales, seed)
    lm, am = lm.to(dtype), am.to(dtype)
    ref = lattices(lm.double(), am.double(), symbols, rnnt_type, scales, seed)
    for a, b in zip(got[:2], ref[:2]):
        fin = torch.isfinite(b)
        assert torch.equal(torch.isfinite(a), fin)
        assert float(((a.double() - b).abs() - 1e-6 * b.abs())[fin].max()) < 1e-5
    eps = 2e-5 if dtype == torch.float32 else float(torch.finfo(dtype).eps)
    for a, b in zip(got[2:], ref[2:]):
        assert float((a.double() - b).norm()) < eps * float(b.norm())


@pytest.mark.parametrize("rnnt_type", ["regular", "modified", "constrained"])
@pytest.mark.parametrize("C", [51, 52, 500, 501, 4233])
@pytest.mark.parametrize("sigma", [2.0, 4.0, 6.0, 10.0])
def test_spread_logits(sigma, C, rnnt_type):
    B, S, T = 2, 41, 70
    torch.manual_seed(C)
    lm, am = sigma * torch.randn(B, S + 1, C).cuda(), sigma * torch.randn(B, T, C).cuda()
    am[:, ::3] *= 0.1  # flat frames beside the peaked ones
    symbols = torch.randint(1, C, (B, S)).cuda()
    for scales in ((0.0, 0.0), (0.25, 0.0), (0.25, 0.1)):
        check(lm, am, symbols, rnnt_type, scales, C)


@pytest.mark.parametrize("rnnt_type", ["regular", "constrained"])
@pytest.mark.parametrize("C", [51, 52, 501])
@pytest.mark.parametrize("peak", [15.0, 20.0, 30.0, 60.0])
def test_rows_that_peak_at_different_symbols(peak, C, rnnt_type):
    B, S, T = 2, 33, 40
    torch.manual_seed(C)
    symbols = torch.randint(1, C, (B, S)).cuda()
    lm, am = torch.zeros(B, S + 1, C).cuda(), torch.zeros(B, T, C).cuda()
    lm[..., 3] = peak
    am[..., 5] = peak
    for scales in ((0.0, 0.0), (0.25, 0.1)):
        check(lm, am, symbols, rnnt_type, scales, C)
    # one such row and one such frame in an ordinary utterance
    lm, am = torch.randn(B, S + 1, C).cuda(), torch.randn(B, T, C).cuda()
    lm[0, 7] = 0
    lm[0, 7, 3] = peak
    am[0, 11] = 0
    am[0, 11, 5] = peak
    for scales in ((0.0, 0.0), (0.25, 0.1)):
        check(lm, am, symbols, rnnt_type, scales, C)


@pytest.mark.parametrize("S,T", [(127, 140), (128, 33), (200, 210), (8, 257)])
def test_weak_cells_at_the_edges_of_tiles(S, T):
    B, C = 2, 37
    torch.manual_seed(S)
    lm, am = torch.randn(B, S + 1, C).cuda(), torch.randn(B, T, C).cuda()
    for s in {0, S // 2, min(S, 31), min(S, 32), min(S, 127), S}:
        lm[:, s] = 0
        lm[:, s, 3] = 40
    for t in (0, T // 2, T - 1):
        am[:, t] = 0
        am[:, t, 5] = 40
    symbols = torch.randint(1, C, (B, S)).cuda()
    for rnnt_type in ("regular", "modified", "constrained") if T >= S else ("regular",):
        check(lm, am, symbols, rnnt_type, (0.25, 0.1), S)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("C", [52, 501])
def test_16_bit_inputs(C, dtype):
    torch.manual_seed(C)
    lm, am = 6 * torch.randn(2, 20, C).cuda(), 6 * torch.randn(2, 40, C).cuda()
    symbols = torch.randint(1, C, (2, 19)).cuda()
    check(lm, am, symbols, "regular", (0.25, 0.0), C, dtype)


@pytest.mark.parametrize("C", [51, 52])
def test_symbols_that_are_improbable_in_every_row(C):
    """The unigram of a target symbol down to e^-40: its share of the am-only gradient is O(1)."""
    torch.manual_seed(C)
    lm, am = torch.randn(2, 20, C).cuda(), torch.randn(2, 40, C).cuda()
    lm[..., 7] -= 40
    am[:, 3:6] = 0
    am[:, 3:6, 7] = 50
    symbols = torch.full((2, 19), 7).cuda()
    check(lm, am, symbols, "regular", (0.25, 0.1), C)


@pytest.mark.parametrize("C", [51, 52])
def test_beyond_the_range_of_float32(monkeypatch, C):
    """Peaks of 100 nats: float32 sums end at the smallest normal number, as on the FMA pipe."""
    torch.manual_seed(C)
    lm, am = torch.zeros(2, 20, C).cuda(), torch.zeros(2, 40, C).cuda()
    lm[..., 3] = 100
    am[..., 5] = 100
    symbols = torch.randint(1, C, (2, 19)).cuda()
    got = lattices(lm, am, symbols, "regular", (0.0, 0.0), C)
    monkeypatch.setenv("FRNNT_CONTRACTION", "simt")
    ref = lattices(lm, am, symbols, "regular", (0.0, 0.0), C)
    for a, b in zip(got, ref):
        torch.testing.assert_close(a, b, rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("C", [51, 52])
@pytest.mark.parametrize("weight", [1e10, float("inf"), float("nan")])
@pytest.mark.parametrize("peaked", [False, True])
def test_gradients_do_not_depend_on_the_other_utterances(C, weight, peaked):
    import fast_rnnt_b200 as fr
    torch.manual_seed(C)
    lm, am = torch.randn(3, 21, C).cuda(), torch.randn(3, 40, C).cuda()
    symbols = torch.randint(1, C, (3, 20)).cuda()
    if peaked:
        lm[1], am[1] = 0, 0
        lm[1, :, 3], am[1, :, 5] = 20, 20
    lm.requires_grad_(True)
    am.requires_grad_(True)
    px, py = fr.get_rnnt_logprobs(lm, am, symbols, 0)
    gx, gy = torch.rand_like(px), torch.rand_like(py)
    alone = torch.autograd.grad([px, py], [lm, am], [gx, gy], retain_graph=True)
    gx[1] *= weight
    gy[1] *= weight
    beside = torch.autograd.grad([px, py], [lm, am], [gx, gy])
    for a, b in zip(alone, beside):
        assert torch.equal(a[0], b[0]) and torch.equal(a[2], b[2])


@pytest.mark.parametrize("C", [51, 52])
@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan")])
def test_a_cell_without_a_finite_gradient_spoils_its_row_and_frame_only(C, value):
    import fast_rnnt_b200 as fr
    torch.manual_seed(C)
    lm = torch.randn(1, 21, C).cuda().requires_grad_(True)
    am = torch.randn(1, 40, C).cuda().requires_grad_(True)
    px, py = fr.get_rnnt_logprobs(lm, am, torch.randint(1, C, (1, 20)).cuda(), 0)
    gx, gy = torch.rand_like(px) * 1e-3, torch.rand_like(py) * 1e-3
    alone = torch.autograd.grad([px, py], [lm, am], [gx, gy], retain_graph=True)
    gx[0, 4, 7] = value
    beside = torch.autograd.grad([px, py], [lm, am], [gx, gy])
    for a, b, i in zip(alone, beside, (4, 7)):
        others = [k for k in range(a.shape[1]) if k != i]
        torch.testing.assert_close(a[0, others], b[0, others], rtol=1e-6, atol=1e-9)
        assert not torch.isfinite(b[0, i]).all()
