"""Out of host memory inside a C entry: it answers with an error, it neither
throws nor ends the process.  In a child process whose address space is capped
a little above what it holds, over caps that end the build of the row-segment
stream at each of its allocations."""
import os
import pathlib
import subprocess
import sys

REPO = pathlib.Path(__file__).resolve().parent.parent

CHILD = """
import resource, sys
import numpy as np
sys.path.insert(0, sys.argv[1])
import cbspmv
from cbspmv import gen
n, per = 30000, 12
rng = np.random.default_rng(1)
cols = np.sort(rng.integers(0, n, (n, per)) // per * per + np.arange(per), axis=1) % n
coo = gen.Coo(n, n, np.repeat(np.arange(n), per).astype(np.int32),
              np.sort(cols, axis=1).reshape(-1).astype(np.int32), rng.standard_normal(n * per))
plan = cbspmv.Plan(coo)
name = b"rs_sizes:4736"
export = cbspmv.lib().cbspmv_export
assert export(plan._h, name, None) == 6
hard = resource.getrlimit(resource.RLIMIT_AS)[1]
got = []
for k in range(160):
    size = int(open("/proc/self/statm").read().split()[0]) * resource.getpagesize()
    resource.setrlimit(resource.RLIMIT_AS, (size + (k << 18), hard))
    got.append(export(plan._h, name, None))
    resource.setrlimit(resource.RLIMIT_AS, (hard, hard))
assert set(got) == {-1, 6}, got
assert export(plan._h, name, None) == 6
print("fine", got.count(-1))
"""


def test_stream_build_out_of_memory():
    env = dict(os.environ, OMP_NUM_THREADS="1", MALLOC_TOP_PAD_="0")
    r = subprocess.run([sys.executable, "-c", CHILD, str(REPO / "cb-sparse-dcu_b200")], env=env,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.startswith("fine"), (r.returncode, r.stderr[-2000:])
