"""First pairs dealt over the blocks, the rest handed out by the counter: sets of
a pair per group of a full launch, one more and one less, and a few more rounds,
against the oracle."""
import numpy as np
import pytest
import torch

import oracle as O
from ish_gb300 import native
from test_gpu_parity import THREADS, assert_same, ctx  # noqa: F401
from test_gpu_small_sets import make_query, random_set

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("G", [1, 8, 32])
@pytest.mark.parametrize("algo", [native.ALGO_SEMI_GLOBAL, native.ALGO_LOCAL])
def test_pairs_per_group(ctx, G, algo):  # noqa: F811
    rng = np.random.default_rng(G)
    groups = torch.cuda.get_device_properties(0).multi_processor_count * 512 // G
    K = -(-24 // G)
    ctx.set_option(native.OPT_WAVE_GROUP, G)
    ctx.set_option(native.OPT_WAVE_K, K)
    try:
        qid, om = make_query(ctx, rng.integers(0, 4, G * K - 1, dtype=np.uint8), algo)
        for n in (2 * groups - 1, 2 * groups, 2 * groups + 1, 5 * groups):
            buf, off = random_set(rng, n, 900)
            assert_same(ctx.score(qid, buf, off), om.batch(buf, off, threads=THREADS), f"G={G} n={n}")
        ctx.free_query(qid)
    finally:
        ctx.set_option(native.OPT_WAVE_GROUP, 0)
        ctx.set_option(native.OPT_WAVE_K, 0)
