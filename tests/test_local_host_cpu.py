"""Host side of the one-rank paths (csrc/bindings_local.cpp) that needs no GPU."""
import os
import subprocess
import sys

import torch

from teramoe_b200.parallel import world as world_module
from teramoe_b200.parallel.world import EPWorld

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


class _Arena:
    def __init__(self, log, name):
        self.log, self.name = log, name

    def local_ptr(self):
        return 4096 * self.name

    def close(self):
        self.log.append(("free", self.name))


def _logged_world(monkeypatch):
    log, names = [], iter(range(1, 9))
    w = EPWorld.single("cpu")
    monkeypatch.setattr(world_module.torch.cuda, "synchronize", lambda device=None: log.append(("wait",)))
    monkeypatch.setattr(w, "_new_arena", lambda n: _Arena(log, next(names)))
    monkeypatch.setattr(w, "_open_ipc", lambda arena: None)
    w.on_arena_change = lambda ptr, n: log.append(("use", ptr // 4096))
    return w, log


def test_an_arena_is_freed_behind_a_wait_for_its_last_user(monkeypatch):
    """A backward pass in another thread may launch on the old arena until it is told of the new one: the wait that the old one is
    freed behind comes after that."""
    w, log = _logged_world(monkeypatch)
    w.ensure_data(1000)
    w.ensure_data(5000)
    w.ensure_data(10)
    assert [e for e in log if e[0] != "wait"] == [("use", 1), ("use", 2), ("free", 1)]
    told, freed = log.index(("use", 2)), log.index(("free", 1))
    assert ("wait",) in log[told:freed]


def test_closing_a_world_takes_the_arena_away_before_it_waits(monkeypatch):
    w, log = _logged_world(monkeypatch)
    w.ensure_data(1000)
    w.is_cuda, w.control = True, _Arena(log, 8)
    monkeypatch.setattr(w, "check_status", lambda: None)
    w.close()
    taken = log.index(("use", 0))
    assert ("wait",) in log[taken:log.index(("free", 1))]


def test_the_native_layer_follows_the_arena():
    from teramoe_b200._build import load_ext
    layer = load_ext().LocalLayer(torch.zeros(8, dtype=torch.int32), torch.zeros(4, dtype=torch.int32))
    layer.set_arena(4096, 100)
    assert layer.arena() == 4096


def test_a_build_is_recognised_by_the_next_process(monkeypatch, tmp_path):
    """The stamp of a build is the hash that another process computes from the same sources and flags, whatever the build does with them."""
    from torch.utils import cpp_extension

    from teramoe_b200 import _build
    monkeypatch.setattr(_build, "_EXT_DIR", tmp_path)
    monkeypatch.setattr(cpp_extension, "load", lambda **kw: [kw[k].append("-more") for k in ("extra_cflags", "extra_cuda_cflags", "extra_ldflags")])
    before = _build._source_hash()
    _build.build()
    assert _build._stamp_path().read_text() == before == _build._source_hash()


def test_rows_of_the_second_cta_are_published_at_cluster_scope():
    """The loading warps' arrive is all that orders the second CTA's rows before the products that the first one issues.  A missing order
    shows on the GPU rarely or never, so what is looked at is the source: the arrive from the second CTA and every wait of the issuer for a
    stage that such rows may fill are a release and an acquire at cluster scope."""
    src = open(os.path.join(ROOT, "teramoe_b200", "csrc", "local_layer.cu")).read()
    hand_over = src[src.index("auto hand_over = "):]
    hand_over = hand_over[: hand_over.index("};")]
    assert "mbar_arrive_cluster_release" in hand_over and "mbar_arrive_cluster(" not in hand_over
    issuer = src[src.index("// ----", src.index("TMA producer")):]
    issuer = issuer[issuer.index("UMMA issuer"): issuer.index("epilogue, then gather")]
    waits = [line for line in issuer.splitlines() if "mbar_wait" in line and "full_bar" in line and "tfull_bar" not in line]
    assert waits and all("mbar_wait_cluster_acquire" in line for line in waits)


def test_kernels_of_a_call_by_its_sizes():
    """A forward with few rows per expert gathers its rows from x: no memory for copies of them, whatever I is."""
    from teramoe_b200._build import load_ext
    variant = lambda T, K, E, I, keep: tuple(int(v) for v in load_ext().local_layer_variant(T, K, E, 4096, I, keep).values())
    assert variant(8, 2, 8, 4096, False) == (1, 0, 0)
    assert variant(64, 2, 8, 14336, False) == (1, 0, 0)
    assert variant(65, 2, 8, 14336, False) == (0, 1, 0)
    assert variant(64, 2, 9, 14336, False) == (1, 0, 0)
    assert variant(128, 2, 16, 14336, False) == (1, 0, 0)
    assert variant(129, 2, 17, 14336, False) == (2, 1, 0)       # (the routing decides: both kernels are launched)
    assert variant(192, 2, 24, 1024, False) == (1, 0, 0)        # (four units read again, 96 MB)
    assert variant(193, 2, 25, 1024, False) == (2, 0, 0)
    assert variant(512, 2, 8, 4032, False) == (0, 0, 0)
    assert variant(8, 2, 8, 14336, True) == (0, 1, 1)
    assert variant(511, 2, 4, 512, True) == (0, 0, 1)
    assert variant(512, 2, 4, 512, True) == (0, 0, 0)
    assert variant(0, 2, 4, 512, False) == (0, 0, 0)


def test_which_forwards_have_few_rows_per_expert():
    """Up to 16 rows on average; where I is below 4096 up to 40 and I / 10, up to 64 and I / 32, and with 128 tokens at most up to 80."""
    from teramoe_b200._build import load_ext
    few = lambda T, K, E, I: load_ext().local_layer_variant(T, K, E, 4096, I, False)["few"]
    assert [few(T, 2, 8, 256) for T in (64, 65, 128)] == [1, 1, 1]
    assert [few(T, 2, 16, 256) for T in (128, 129, 204, 205)] == [1, 2, 2, 0]
    assert [few(T, 2, 8, 4032) for T in (128, 129, 256, 257)] == [1, 2, 2, 0]
    assert [few(T, 2, 8, 1536) for T in (160, 161, 192, 193)] == [2, 2, 2, 0]
    assert [few(T, 6, 8, 64) for T in (106, 107)] == [1, 0]
    assert [few(T, 2, 8, 4096) for T in (64, 65)] == [1, 0]
    assert few(128, 8, 8, 4032) == 0
    assert load_ext().local_layer_variant(128, 2, 8, 4096, 4032, True)["few"] == 0
