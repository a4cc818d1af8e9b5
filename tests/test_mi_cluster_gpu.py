"""The float lattice sweeps (csrc/mi_f32.cu) at the sizes where their split changes: one row per
lane up to 32 lattice rows, two up to 64, a cluster of 2 .. 8 CTAs up to 512, row blocks
beyond; chunks of 16 diagonals.  Tolerances are those of test_mi_gpu.py."""
import random

import pytest
import torch

from oracle import rnnt_oracle as orc
from tests import workloads
from tests.test_mi_gpu import assert_close

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (31, 16), (32, 17), (63, 15), (64, 97), (127, 130), (128, 144), (191, 200), (383, 40),
         (511, 33), (512, 20), (1024, 50)]


def run(px, py, bnd, w):
    from fast_rnnt_b200 import mutual_information as mi
    cb = None if bnd is None else bnd.cuda()
    ans, _, lattice = mi.mi_forward(px.cuda(), py.cuda(), cb)
    gx, gy = mi.mi_backward_from_lattice(px.cuda(), lattice, cb, w.cuda(), py.shape)
    return ans.cpu(), gx.cpu(), gy.cpu()


@pytest.mark.parametrize("modified", [False, True])
@pytest.mark.parametrize("S,T", SIZES)
def test_sweeps_at_the_edges_of_their_split(S, T, modified):
    rng = random.Random(S)
    torch.manual_seed(S + T)
    B, T = 3, max(T, S) if modified else T
    px = torch.rand(B, S, T + (0 if modified else 1)) * -4
    py = torch.rand(B, S + 1, T) * -4
    w = torch.linspace(0.5, 1.5, B)
    for bnd in (None, workloads.random_mi_boundary(B, S, T, modified, rng)):
        p, ans = orc.mi_forward_raw(px, py, bnd)
        gx, gy = orc.mi_backward_raw(px, py, bnd, p, w)
        got = run(px, py, bnd, w)
        assert_close(got[0], ans, 1e-6, 1e-4, "ans")
        # a chain of S + T cells of rounding up to 1e-4 each near a score of -2000
        tol = 2e-5 if S + T < 700 else 1e-4
        assert_close(got[1], gx, 0, tol, "px_grad")
        assert_close(got[2], gy, 0, tol, "py_grad")


@pytest.mark.parametrize("modified", [False, True])
@pytest.mark.parametrize("S,T", [(20, 50), (40, 60), (100, 120)])
def test_special_values_as_the_row_per_thread_sweeps(monkeypatch, S, T, modified):
    torch.manual_seed(S)
    lowest = torch.finfo(torch.float32).min
    specials = [float("-inf"), float("inf"), float("nan"), lowest, -1e30, -1e6]
    B = 2 * len(specials)
    px = torch.rand(B, S, T + (0 if modified else 1)) * -4
    py = torch.rand(B, S + 1, T) * -4
    for i, v in enumerate(specials):
        px[2 * i, S // 2, T // 3] = v
        py[2 * i, S // 3, T // 2] = v
        px[2 * i + 1, S // 2] = v      # every path meets it
    w = torch.ones(B)
    got = run(px, py, None, w)
    monkeypatch.setenv("FRNNT_MI", "row_per_thread")
    ref = run(px, py, None, w)
    for a, b, what in zip(got, ref, ("ans", "px_grad", "py_grad")):
        assert torch.equal(torch.isnan(a), torch.isnan(b)), what
        a, b = torch.nan_to_num(a, nan=0.0), torch.nan_to_num(b, nan=0.0)
        assert_close(a, b, 2e-6, 2e-5, what)


@pytest.mark.parametrize("S,T", [(20, 40), (100, 70)])
def test_scratch_off_a_16_byte_boundary(S, T):
    """Both families of float sweeps keep the same scratch: an unaligned copy takes the other one."""
    from fast_rnnt_b200 import mutual_information as mi
    torch.manual_seed(S)
    px, py = (torch.rand(2, S, T + 1) * -4).cuda(), (torch.rand(2, S + 1, T) * -4).cuda()
    w = torch.ones(2).cuda()
    _, _, lattice = mi.mi_forward(px, py, None)
    moved = torch.empty(lattice.numel() + 4, dtype=torch.uint8, device="cuda")[4:]
    moved.copy_(lattice)
    for a, b in zip(mi.mi_backward_from_lattice(px, lattice, None, w, py.shape),
                    mi.mi_backward_from_lattice(px, moved, None, w, py.shape)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("modified", [False, True])
@pytest.mark.parametrize("S,T", [(40, 60), (64, 70), (100, 120), (300, 330), (600, 640)])
def test_a_wait_that_runs_out_shows(S, T, modified):
    """With no patience at all for the row of the CTA above (below), whatever depends on it is NaN:
    the lattice from row 64 on and the score, resp. the gradients of the rows above the last CTA's and
    what reaches the origin.  Nothing hangs, and the next call is right."""
    from fast_rnnt_b200 import _lib
    from fast_rnnt_b200._lib import ptr
    torch.manual_seed(S)
    B = 3
    px = (torch.rand(B, S, T + (0 if modified else 1)) * -4).cuda()
    py = (torch.rand(B, S + 1, T) * -4).cuda()
    w = torch.ones(B).cuda()

    def sweeps(forward_tries, backward_tries):
        lattice = torch.zeros(_lib.lib().frnnt_mi_lattice_bytes(0, B, S, T), dtype=torch.uint8, device="cuda")
        p = torch.zeros(B, S + 1, T + 1).cuda()
        ans, origin = torch.zeros(B).cuda(), torch.zeros(B).cuda()
        gx, gy = torch.zeros_like(px), torch.zeros_like(py)
        _lib.call("frnnt_mi_sweeps_limited", ptr(px), ptr(py), None, ptr(w), ptr(p), ptr(ans), ptr(gx), ptr(gy),
                  ptr(origin), ptr(lattice), B, S, T, int(modified), forward_tries, backward_tries,
                  _lib.stream_ptr(px.device))
        torch.cuda.synchronize()
        return p, ans, gx, gy, origin

    good = sweeps(-1, -1)
    reachable = torch.isfinite(good[0])
    assert reachable[:, S, T].all()
    p, ans, _, _, _ = sweeps(0, -1)
    _, _, gx, gy, origin = sweeps(-1, 0)
    if S + 1 <= 64:   # one CTA
        assert torch.equal(p, good[0]) and torch.equal(gx, good[2]) and torch.equal(gy, good[3])
    else:
        assert torch.equal(p[:, :64], good[0][:, :64])
        assert torch.isnan(p[:, 64:][reachable[:, 64:]]).all() and torch.isnan(ans).all()
        last = S // 64 * 64   # first row of the CTA that waits for nobody
        assert torch.equal(gy[:, last:], good[3][:, last:])
        # (modified: a cell too late to reach that row depends on nothing there; its gradient is 0)
        assert torch.isnan(gy[:, :last][good[3][:, :last] != 0]).all() and torch.isnan(origin).all()
        assert torch.isnan(gx[:, :last - 1][good[2][:, :last - 1] != 0]).all()
    for a, b in zip(sweeps(-1, -1), good):
        assert torch.equal(a, b)


@pytest.mark.parametrize("modified", [False, True])
@pytest.mark.parametrize("S,T", [(31, 60), (63, 70), (100, 130), (200, 210), (511, 530), (600, 620)])
def test_bit_for_bit_as_the_row_per_thread_sweeps(monkeypatch, S, T, modified):
    """expf and log1pf in the same order: prune ranges, an argmax, move with the last bit."""
    torch.manual_seed(S)
    rng = random.Random(S)
    B = 4
    px = torch.rand(B, S, T + (0 if modified else 1)) * -4
    py = torch.rand(B, S + 1, T) * -4
    for bnd in (None, workloads.random_mi_boundary(B, S, T, modified, rng)):
        got = run(px, py, bnd, torch.linspace(0.5, 1.5, B))
        monkeypatch.setenv("FRNNT_MI", "row_per_thread")
        ref = run(px, py, bnd, torch.linspace(0.5, 1.5, B))
        monkeypatch.delenv("FRNNT_MI")
        for a, b in zip(got, ref):
            assert torch.equal(a, b)
