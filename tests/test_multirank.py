"""Host logic of multi-GPU runs, on CPU with two gloo ranks: bench.py's
replicas report the slowest rank's time on every rank, and the ranks other
than 0 of the reference arm exit without output (rank 0 alone runs and prints
the CPU baseline); the arm's line where the reference is not built."""
from __future__ import annotations

import json
import os
import socket
import subprocess
import sys

import torch.multiprocessing as mp

from conftest import ROOT


def _free_port() -> int:
    with socket.socket() as s:
        s.bind(("127.0.0.1", 0))
        return s.getsockname()[1]


def _rank(rank: int, port: int, out):
    import datetime

    import torch.distributed as dist
    sys.path.insert(0, str(ROOT))
    import bench
    dist.init_process_group("gloo", init_method=f"tcp://127.0.0.1:{port}", rank=rank, world_size=2,
                            timeout=datetime.timedelta(seconds=60))
    t = bench.max_over_ranks(1.5 + rank, 2, device="cpu")
    dist.barrier()
    out[rank] = t
    dist.destroy_process_group()


def test_max_over_ranks_gloo():
    port = _free_port()
    ctx = mp.get_context("spawn")
    with ctx.Manager() as m:
        out = m.dict()
        procs = [ctx.Process(target=_rank, args=(r, port, out)) for r in range(2)]
        for p in procs:
            p.start()
        for p in procs:
            p.join(120)
            assert p.exitcode == 0
        assert dict(out) == {0: 2.5, 1: 2.5}


def test_reference_arm_other_ranks_exit_quietly():
    env = dict(os.environ, RANK="1", WORLD_SIZE="2", LOCAL_RANK="1")
    r = subprocess.run([sys.executable, str(ROOT / "bench.py"), "--impl", "reference", "--steps", "3"],
                       env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0
    assert r.stdout.strip() == ""


def test_reference_arm_without_the_reference(monkeypatch, capsys):
    """A machine without the library built from the reference's sources: one line that says so, exit code 0."""
    import bench
    from oracle import ref
    monkeypatch.setattr(ref, "LIB", ROOT / "oracle" / "_ref" / "absent.so")
    monkeypatch.setattr(sys, "argv", ["bench.py", "--impl", "reference"])
    for k in ("RANK", "WORLD_SIZE", "LOCAL_RANK"):
        monkeypatch.delenv(k, raising=False)
    assert bench.main() == 0
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and line["unavailable"]
