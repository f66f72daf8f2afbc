"""What the launchers decide on the host before anything is launched: no GPU is needed."""
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_a_product_of_no_groups_launches_nothing():
    """(In a process of its own: it used to end with a division by zero.)"""
    code = ("import torch\nfrom moe_b200.ops import core\nL = core.lib()\n"
            "buf = torch.zeros(64)\np = buf.data_ptr() + (-buf.data_ptr()) % 16\n"
            "assert L.moe_gemm_generic(p, 0, 4, None, 5, p, 0, 32, p, 0, 8, None, p, 0, 5, 8, 4, p, None, 0, None) == 0\n")
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True)
    assert r.returncode == 0, (r.returncode, r.stderr[-500:])


def test_pairs_of_ctas_are_for_plain_products_of_many_rows():
    from moe_b200.ops import tc

    pairs = tc.lib().moe_gemm_tc_pairs
    assert [pairs(m, 0, 0) for m in (2048, 3071, 3072, 100000)] == [0, 0, 1, 1]
    assert [pairs(60 * m, 60, 0) for m in (137, 255, 256, 546)] == [0, 0, 1, 1]
    assert not any(pairs(m, g, 1) for m in (4096, 8192, 100000) for g in (0, 4, 16))          # gate and up rows share a tile: nothing to gain
