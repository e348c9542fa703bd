"""The autotuner's choice and its cache, with a context that only times."""
import json
from types import SimpleNamespace

from gsofa_b200 import autotune


class _Timed:
    """symbfact_batch of this context takes as long as `ms` says."""

    def __init__(self, ms):
        self.ms = ms
        self.runs = []

    def symbfact_batch(self, mats, p):
        c = (p.block_size, p.threads_per_source, p.src_chunk)
        self.runs.append(c)
        return [SimpleNamespace(kernel_ms=self.ms(c))]


MATS = [SimpleNamespace(n=5000, nnz=25000), SimpleNamespace(n=900, nnz=4000)]


def test_candidates_differ_in_what_they_run():
    # threads_per_source chooses nothing
    assert len({(b, chunk) for b, _, chunk in autotune.DEFAULT_CANDIDATES}) == len(autotune.DEFAULT_CANDIDATES)


def test_a_choice_of_former_kernels_is_measured_anew(tmp_path):
    path = tmp_path / "tune.json"
    key = autotune.signature(MATS)
    path.write_text(json.dumps({key: {"choice": [1024, 1, 512], "kernel_ms": 1.0},
                                "n1-nnz1-k1": {"choice": [256, 1, 0], "kernel_ms": 2.0}}))
    ctx = _Timed(lambda c: 1.0 if c == (0, 1, 0) else 2.0)
    best, rep = autotune.autotune(ctx, MATS, cache_path=str(path))
    assert not rep["cached"] and rep["choice"] == [0, 1, 0]
    assert ctx.runs == list(autotune.DEFAULT_CANDIDATES)
    best2, rep2 = autotune.autotune(_Timed(None), MATS, cache_path=str(path))
    assert rep2["cached"] and rep2["choice"] == [0, 1, 0]
    assert (best2.block_size, best2.src_chunk) == (best.block_size, best.src_chunk)
    assert json.loads(path.read_text())["n1-nnz1-k1"]["choice"] == [256, 1, 0]
