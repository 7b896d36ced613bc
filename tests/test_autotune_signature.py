"""A cache of the autotuner names the kernels that it measured: the signature of a
workload changes with their sources, and an entry of other kernels is not applied."""
import json

from starpolymersmd_gb300 import autotune
from tests.test_autotune_cache import FakeContext


def test_signature_follows_the_kernel_sources(tmp_path):
    (tmp_path / "a.cu").write_text("1")
    (tmp_path / "b.cuh").write_text("2")
    first = autotune.kernels_id(str(tmp_path))
    autotune.kernels_id.cache_clear()
    assert autotune.kernels_id(str(tmp_path)) == first
    autotune.kernels_id.cache_clear()
    (tmp_path / "b.cuh").write_text("3")
    assert autotune.kernels_id(str(tmp_path)) != first
    autotune.kernels_id.cache_clear()
    assert autotune.signature(1, 2, 3, 4).endswith("|kernels=" + autotune.kernels_id())


def test_entry_of_other_kernels_is_measured_again(tmp_path):
    path = str(tmp_path / "cache.json")
    key = autotune.signature(1, 80000, 8000, 121)
    old = key[:key.index("|kernels=")]  # what a cache held before it named the kernels
    with open(path, "w") as f:
        json.dump({old: {"index": [0, 5, 4, 0], "report": {}}}, f)
    ctx = FakeContext(tuned=(1, 0, 0), pmd=0)
    assert autotune.tune(ctx, key, cache_path=path)["cached"] is False
    assert ctx.get_variants() == (1, 0, 0)
