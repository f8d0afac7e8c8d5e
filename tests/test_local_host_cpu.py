"""Host side of the one-rank paths (csrc/bindings_local.cpp) that needs no GPU."""
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _python(code: str) -> str:
    """Output of a child process: what is tested here ended the process when it went wrong."""
    env = dict(os.environ, PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300, env=env)
    assert r.returncode == 0, f"exit code {r.returncode}\n{r.stdout}\n{r.stderr}"
    return r.stdout


def test_a_reported_wait_is_raised_with_its_numbers():
    out = _python("""
import torch
from teramoe_b200._build import load_ext
status, host = torch.tensor([2, 601, 5, 128, 0, 0, 0, 0], dtype=torch.int32), torch.tensor([2, 601, 5, 128], dtype=torch.int32)
layer = load_ext().LocalLayer(status, host)
try:
    layer.check()
except RuntimeError as e:
    print(str(e).splitlines()[0])
layer.check()
print(status.tolist(), int(host[0]))
""")
    assert "flag wait (site 601, block 5, detail 128)" in out and "[0, 0, 0, 0, 0, 0, 0, 0] 0" in out
