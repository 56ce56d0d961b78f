"""Order of the early-launch instructions in the row kernels, from their source.

F's row kernels (k_row_mul_f, k_grid_mul_f) are launched early and read what the
column passes left before they wait for the kernel ahead of them, G's row
kernel.  That is safe only if G's row kernel allows the launch after its own
wait: an early launch sees an earlier kernel's writes only past a
griddepcontrol.wait, and the column passes are two launches back.
"""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cumodp_b200", "csrc")


def _kernels():
    """name -> body without comments, for every __global__ function of the headers."""
    out = {}
    for f in sorted(os.listdir(CSRC)):
        s = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, f)).read())
        for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\s*\(", s):
            i = s.index("{", m.end())
            depth, j = 1, i + 1
            while depth:
                depth += {"{": 1, "}": -1}.get(s[j], 0)
                j += 1
            out[m.group(1)] = s[i:j]
    return out


def test_g_rows_allow_the_next_launch_only_after_their_wait():
    k = _kernels()
    for g in ("k_row_fwd_g", "k_grid_fwd_g"):
        assert 0 <= k[g].find("pdl_wait()") < k[g].find("pdl_trigger()"), g
    for col in ("k_col_fwd", "k_cold_fwd"):
        # G's rows may then start once these are complete, and not before
        assert "pdl_trigger" not in k[col], col


def test_kernels_that_read_before_their_wait_are_the_known_ones():
    """Every other kernel that is launched early waits before it reads another kernel's words (tables aside)."""
    k = _kernels()
    early = {n for n, b in k.items() if "pdl_wait()" in b}
    assert early == {"k_row_fwd_g", "k_row_mul_f", "k_grid_fwd_g", "k_grid_mul_f", "k_col_inv", "k_cold_inv", "k_lift"}
    for n in ("k_grid_fwd_g", "k_cold_inv", "k_lift", "k_col_inv"):
        before = k[n].split("pdl_wait()")[0]
        assert not re.search(r"__ldg|cp_async|_load|J\.w[ab]\s*\+", before), n
