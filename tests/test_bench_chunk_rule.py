"""The benchmark's roofline counts launches by the library's chunk rule: both state the same
limits."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_benchmark_states_the_librarys_chunk_limits():
    lib = open(os.path.join(ROOT, "eos_b200", "csrc", "wavefront.cu")).read()
    bench = open(os.path.join(ROOT, "bench.py")).read()
    bits = re.search(r"kChunkPathsMax = 1ll << (\d+);", lib).group(1)
    gigs = re.search(r"kQueueBudget = (\d+)ll << 30;", lib).group(1)
    assert f"min(1 << {bits}, ({gigs} << 30) // per_path)" in bench
    assert f"at most 2^{bits} paths" in bench
