"""Simple lattices and their gradients on the tensor-core path for vocabularies that are no
multiple of 4 and for tensors that are not 16-byte aligned, against the float64 path.

The planes carry 22 bits of exp(x - max) in (0, 1], products accumulate in float32: 1e-5 on
the lattices (scores up to 12: an ulp is 1e-6) and 2e-5 of the gradients' norm."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def lattices(lm, am, symbols, rnnt_type, scales, seed):
    import fast_rnnt_b200 as fr
    lm, am = lm.detach().requires_grad_(True), am.detach().requires_grad_(True)
    px, py = fr.get_rnnt_logprobs_smoothed(lm, am, symbols, 0, lm_only_scale=scales[0],
                                           am_only_scale=scales[1], rnnt_type=rnnt_type)
    g = torch.Generator().manual_seed(seed)
    gx = torch.rand(px.shape, generator=g).to(px)
    gy = torch.rand(py.shape, generator=g).to(py)
    gl, ga = torch.autograd.grad([px, py], [lm, am], [gx, gy])
    return px.detach(), py.detach(), gl, ga


@pytest.mark.parametrize("rnnt_type", ["regular", "modified", "constrained"])
@pytest.mark.parametrize("C", [2, 3, 5, 50, 63, 65, 127, 129, 514, 1024, 1025, 2049, 4096, 4233, 8193])
def test_odd_vocabulary_matches_float64(C, rnnt_type):
    B, S, T = 2, 33, 131
    torch.manual_seed(C)
    lm, am = torch.randn(B, S + 1, C).cuda(), torch.randn(B, T, C).cuda()
    symbols = torch.randint(1, C, (B, S)).cuda()
    for scales in ((0.0, 0.0), (0.25, 0.1)):
        got = lattices(lm, am, symbols, rnnt_type, scales, C)
        ref = lattices(lm.double(), am.double(), symbols, rnnt_type, scales, C)
        for a, b in zip(got[:2], ref[:2]):
            fin = torch.isfinite(b)
            assert torch.equal(torch.isfinite(a), fin)
            assert float((a.double() - b)[fin].abs().max()) < 1e-5
        for a, b in zip(got[2:], ref[2:]):
            assert float((a.double() - b).norm()) < 2e-5 * float(b.norm())


@pytest.mark.parametrize("C", [64, 65])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
def test_unaligned_tensors(C, dtype):
    B, S, T = 2, 9, 40
    torch.manual_seed(C)
    lm, am = torch.randn(B, S + 1, C).to(dtype).cuda(), torch.randn(B, T, C).to(dtype).cuda()
    symbols = torch.randint(1, C, (B, S)).cuda()

    def shifted(x):
        flat = torch.empty(x.numel() + 1, dtype=x.dtype, device=x.device)
        flat[1:] = x.reshape(-1)
        return flat[1:].view(x.shape)

    got = lattices(shifted(lm), shifted(am), symbols, "regular", (0.25, 0.0), C)
    ref = lattices(lm.double(), am.double(), symbols, "regular", (0.25, 0.0), C)
    for a, b in zip(got[:2], ref[:2]):
        fin = torch.isfinite(b)
        assert torch.equal(torch.isfinite(a), fin)
        assert float((a.double() - b)[fin].abs().max()) < 1e-5
    eps = 2e-5 if dtype == torch.float32 else float(torch.finfo(dtype).eps)
    for a, b in zip(got[2:], ref[2:]):
        assert float((a.double() - b).norm()) < eps * float(b.norm())


def off_by_one(x):
    flat = torch.empty(x.numel() + 1, dtype=x.dtype, device=x.device)
    flat[1:] = x.reshape(-1)
    return flat[1:].view(x.shape)


@pytest.mark.parametrize("C", [128, 500])
def test_unaligned_float32_keeps_float32_accuracy(C):
    """Rounding px (about -8 here) to float32 alone is 5e-8 of its norm; sums in groups of 128 values are
    off by 1.2e-7 and more, float32 sums by 6e-8 at most.  Gradients likewise."""
    torch.manual_seed(C)
    lm, am = torch.randn(4, 41, C).cuda(), torch.randn(4, 160, C).cuda()
    symbols = torch.randint(1, C, (4, 40)).cuda()
    got = lattices(off_by_one(lm), off_by_one(am), symbols, "modified", (0.0, 0.0), C)
    ref = lattices(lm.double(), am.double(), symbols, "modified", (0.0, 0.0), C)
    for a, b, bound in zip(got, ref, (8e-8, 8e-8, 8e-8, 9e-8)):
        assert float((a.double() - b).norm()) < bound * float(b.norm())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_unaligned_16_bit_rows_equal_their_float32_copies(dtype):
    torch.manual_seed(0)
    C = 64
    lm, am = torch.randn(2, 10, C).to(dtype).cuda(), torch.randn(2, 40, C).to(dtype).cuda()
    symbols = torch.randint(1, C, (2, 9)).cuda()
    got = lattices(off_by_one(lm), off_by_one(am), symbols, "regular", (0.25, 0.0), C)
    ref = lattices(lm.float(), am.float(), symbols, "regular", (0.25, 0.0), C)
    for a, b in zip(got, ref):
        assert torch.equal(a, b.to(a.dtype))


@pytest.mark.parametrize("C", [37, 40])
@pytest.mark.parametrize("offsets", [(4, 0), (0, 4), (4, 4), (16, 16)])
def test_buffers_off_a_16_byte_boundary(C, offsets):
    """The caller's saved area and backward scratch through the C ABI: planes and their tensor maps
    need 16 bytes, other buffers are served in single values."""
    from fast_rnnt_b200 import _lib
    from fast_rnnt_b200._lib import _c_f64, _c_int, _c_vp, ptr
    lib, B, S, T = _lib.lib(), 2, 9, 21
    torch.manual_seed(C)
    lm, am = torch.randn(B, S + 1, C).cuda(), torch.randn(B, T, C).cuda()
    symbols = torch.randint(1, C, (B, S)).cuda()
    gx, gy = torch.rand(B, S, T + 1).cuda(), torch.rand(B, S + 1, T).cuda()
    saved_bytes = lib.frnnt_simple_saved_bytes(0, B, S, T, C)
    scratch_bytes = lib.frnnt_simple_scratch_bytes(0, B, S, T, C)

    def run(off_saved, off_scratch):
        saved = torch.zeros(saved_bytes + 64, dtype=torch.uint8, device="cuda")
        scratch = torch.zeros(scratch_bytes + 64, dtype=torch.uint8, device="cuda")
        sv, sc = _c_vp(saved.data_ptr() + off_saved), _c_vp(scratch.data_ptr() + off_scratch)
        px, py = torch.empty_like(gx), torch.empty_like(gy)
        gl, ga = torch.empty_like(lm), torch.empty_like(am)
        st = _lib.stream_ptr(lm.device)
        _lib.call("frnnt_simple_logprobs_forward", _c_int(0), ptr(lm), ptr(am), ptr(symbols), None, 0, 0, 0,
                  _c_f64(0.0), _c_f64(0.0), _c_f64(0.0), ptr(px), ptr(py), sv, sc, B, S, T, C, st)
        _lib.call("frnnt_simple_logprobs_backward", _c_int(0), ptr(lm), ptr(am), ptr(symbols), None, 0, 0, 0,
                  _c_f64(0.0), _c_f64(0.0), ptr(gx), ptr(gy), sv, sc, ptr(gl), ptr(ga), B, S, T, C, st)
        torch.cuda.synchronize()
        assert not saved[saved_bytes + off_saved:].any() and not scratch[scratch_bytes + off_scratch:].any()
        return px, py, gl, ga

    for a, b in zip(run(*offsets), run(0, 0)):
        torch.testing.assert_close(a, b, rtol=1e-5, atol=1e-5)
