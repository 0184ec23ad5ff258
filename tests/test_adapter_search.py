"""The library's adapter search (esg_pair_adapters: 64 bases compared at once,
base by base for adapters past 64 and codes above the wildcard) against the
oracle's, mate by mate: read and adapter lengths around a word, wildcards in
either, mismatches at the allowance, every overlap at the read's end."""
import os
import subprocess
import sys

import numpy as np
import pytest

from eschalign_b200 import adapter, pack_reads


@pytest.mark.parametrize("alen", [1, 9, 10, 33, 63, 64, 65, 90])
@pytest.mark.parametrize("top", [4, 5, 9])
def test_search_equals_the_oracles(oracle, alen, top):
    rng = np.random.default_rng(alen * 16 + top)
    a1 = rng.integers(0, 4, alen).astype(np.uint8)
    a2 = rng.integers(0, 4, alen).astype(np.uint8)
    if top > 4:
        a1[rng.random(alen) < 0.1] = 4
    mates = []
    for k in range(400):
        n = int(rng.choice([0, 1, 4, 5, 31, 63, 64, 65, 127, 128, 129, 150, 200]))
        r = rng.integers(0, 4, n).astype(np.uint8)
        if n and top > 4:
            r[rng.random(n) < 0.05] = rng.integers(4, top, 1)[0]
        ad = a1 if len(mates) % 2 == 0 else a2
        if n and k % 3:
            at = int(rng.integers(0, n))
            put = ad[:n - at].copy()
            bad = rng.random(put.size) < rng.choice([0.0, 0.05, 0.12])
            put[bad] = (put[bad] + 1) % 4
            r[at:at + put.size] = put
        mates.append(r)
    for mo in (0, 1, 5, 16):
        cfg = dict(r1=a1, r2=a2, min_overlap=mo, max_read_len=0)
        ads, aligned = adapter.pair_adapters(pack_reads(mates), cfg)
        for p in range(len(mates) // 2):
            m1, m2 = mates[2 * p], mates[2 * p + 1]
            want = oracle.pair_adapters(m1, m2, a1, a2, min_overlap=max(mo, 1))
            assert [int(ads[2 * p]), int(ads[2 * p + 1])] == want, (p, mo)
            assert int(aligned[2 * p]) == m1.size - want[0]


def test_search_without_threads_to_be_had():
    """10 000 pairs, which the library shares among threads, in a process with
    no address space left for their stacks: searched on the caller's."""
    code = """
import resource
import numpy as np
from eschalign_b200 import adapter, pack_reads
rng = np.random.default_rng(3)
cfg = adapter.config()
ads = [np.asarray(cfg["r1"], np.uint8), np.asarray(cfg["r2"], np.uint8)]
mates = []
for k in range(20_000):
    r = rng.integers(0, 4, 60).astype(np.uint8)
    at = int(rng.integers(30, 60))
    r[at:] = ads[k % 2][:60 - at]
    mates.append(r)
adapter.pair_adapters(pack_reads(mates[:2]), cfg)  # the library is loaded
mates = pack_reads(mates)
vm = next(int(ln.split()[1]) for ln in open("/proc/self/status") if ln.startswith("VmSize")) << 10
keep = resource.getrlimit(resource.RLIMIT_AS)
resource.setrlimit(resource.RLIMIT_AS, (vm + (1 << 20), keep[1]))
one = adapter.pair_adapters(mates, cfg)
resource.setrlimit(resource.RLIMIT_AS, keep)
two = adapter.pair_adapters(mates, cfg)
assert (one[0] == two[0]).all() and (one[1] == two[1]).all() and one[0].any()
"""
    out = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=120,
                         cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    assert out.returncode == 0, out.stderr[-2000:]
