"""Builds ``libgqa_b200.so`` (and the diagnostics library, the C++ harness and, where torch is installed, the torch
binding) in-tree with nvcc for sm_100a."""
from __future__ import annotations

import importlib.util
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")


def build(target: str = "all", jobs: int | None = None, quiet: bool = True) -> str:
    """Run ``make`` in ``csrc/``; returns the path of the shared library.  ``all`` includes the torch binding where this
    interpreter has torch; the C libraries and the harness need neither."""
    jobs = jobs or max(1, os.cpu_count() or 1)
    targets = [target]
    if target == "all" and importlib.util.find_spec("torch") is not None:
        targets.append("binding")
    for t in targets:
        cmd = ["make", "-C", CSRC, f"-j{jobs}", f"PYTHON={sys.executable}", t]
        out = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
        if out.returncode != 0:
            what = "_gqa_torch.so" if t == "binding" else "libgqa_b200.so"
            raise RuntimeError(f"building {what} failed:\n" + out.stdout[-4000:])
        if not quiet:
            print(out.stdout)
    return os.path.join(HERE, "libgqa_b200.so")


if __name__ == "__main__":
    print(build(quiet=False))
