"""Buffer sizes are remembered by their arguments, so none may depend on an environment switch:
the calls that use the buffers read the switch anew."""
import pytest

SWITCHES = [("FRNNT_PAIR_TILE", "128"), ("FRNNT_CONTRACTION", "tf32"), ("FRNNT_CONTRACTION", "simt"),
            ("FRNNT_MI", "row_per_thread")]

# (B, T, R, S, C, D): partial grad-weight products default / FRNNT_PAIR_TILE=128 on 148 multiprocessors
JOINERS = [(50, 200, 5, 60, 1000, 640),   # 7 / 11
           (64, 400, 5, 60, 5000, 512),   # 11 / 12
           (64, 500, 5, 100, 500, 512),   # 18 / 9
           (2, 33, 5, 12, 500, 512), (3, 50, 4, 20, 128, 64), (3, 50, 4, 20, 100, 512)]


def sizes():
    from fast_rnnt_b200 import _lib
    lib, out = _lib.lib(), []
    for j in JOINERS:
        for what in ("saved", "forward_scratch", "backward_scratch"):
            out.append(getattr(lib, f"frnnt_pruned_joiner_{what}_bytes")(*j))
        B, T, R, S, C, D = j
        out.append(lib.frnnt_matmul_tn_scratch_floats(C, D, B * T * R))
        out.append(lib.frnnt_joiner_input_grads_scratch_bytes(B, T, D))
        for dt in (0, 1):
            out += [lib.frnnt_simple_saved_bytes(dt, B, S, T, C), lib.frnnt_simple_scratch_bytes(dt, B, S, T, C),
                    lib.frnnt_mi_lattice_bytes(dt, B, S, T), lib.frnnt_mi_rows_per_block(dt)]
    return out


@pytest.mark.parametrize("name,value", SWITCHES)
def test_sizes_do_not_depend_on_a_switch(monkeypatch, name, value):
    from fast_rnnt_b200 import build
    build.build()
    for other, _ in SWITCHES:
        monkeypatch.delenv(other, raising=False)
    default = sizes()
    monkeypatch.setenv(name, value)
    assert sizes() == default
