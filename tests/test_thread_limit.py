"""A process that may start no more threads: the work runs on those it has."""
import subprocess
import sys
from pathlib import Path

PKG = Path(__file__).resolve().parent.parent / "g-mm-repair_gb300"

SCRIPT = """
import resource, sys
sys.path.insert(0, sys.argv[1])
import numpy as np
import gmr
want = gmr.gen_mosaic(300, 64, 8, 0.02, 0.002, 3, threads=1).codes()
used = int(open("/proc/self/statm").read().split()[0]) * resource.getpagesize()
resource.setrlimit(resource.RLIMIT_AS, (used + (96 << 20), resource.RLIM_INFINITY))  # room for a few stacks
assert np.array_equal(gmr.gen_mosaic(300, 64, 8, 0.02, 0.002, 3, threads=400).codes(), want)
"""


def test_threads_that_do_not_start():
    r = subprocess.run([sys.executable, "-c", SCRIPT, str(PKG)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
