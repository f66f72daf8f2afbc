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
