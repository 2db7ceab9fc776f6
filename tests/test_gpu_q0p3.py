"""q0 = 2^64 - 2^32 + 1 with p3 = 3 2^30 + 1: the primes of products of more
than 2^29 coefficients, of served requests and cyclic products above the
31-bit primes' lengths, and of every product with GBNTT_P31=0. The tests of
batches, wave graphs, the serving loop, the radix-3 stage and the prime sets,
which otherwise run on the 31-bit primes, once more on these."""
import os

import numpy as np
import pytest

from cryptography_gb300 import cudart, synth
from test_gpu_batch import (test_batch_empty_and_all_max, test_batch_many_tiny_products_on_a_small_engine,  # noqa: F401
                            test_batch_mixed_sizes_match_single, test_batch_multi_wave_bucket,
                            test_batch_pairs_sharing_right_operand, test_batch_shared_right_operand,
                            test_batch_uneven_products_split)
from test_gpu_graphs import (test_mixed_bucket_batches_replay, test_plan_change_drops_graphs,  # noqa: F401
                             test_replayed_waves_match_single_products)
from test_gpu_primes import (test_batched_two_prime_matches_single, test_engine_knobs_give_identical_products,  # noqa: F401
                             test_largest_coefficients, test_sets_agree_at_length_boundaries,
                             test_squares_and_random_sizes)
# (the default threshold's test first: it needs the engine without r3engine's)
from test_gpu_radix3 import (test_radix3_default_threshold, r3engine, test_radix3_all_max_and_squares,  # noqa: F401
                             test_radix3_batch_one_size, test_radix3_batches, test_radix3_device_pointers_and_aliasing,
                             test_radix3_lengths_match_oracle, test_radix3_path_is_taken,
                             test_radix3_pinned_host_operands, test_radix3_shared_and_paired_waves_alone)
from test_gpu_serving import test_serving_mix_equals_alone, test_serving_radix3_requests  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def engine(engine):
    old = os.environ.get("GBNTT_P31")
    os.environ["GBNTT_P31"] = "0"
    engine.teardown()
    try:
        engine.init(24)
        yield engine
    finally:
        if old is None:
            del os.environ["GBNTT_P31"]
        else:
            os.environ["GBNTT_P31"] = old
        engine.teardown()
        engine.init(24)


def _launches(engine, na, nb):
    a, b, c = (cudart.DeviceBuffer(4 * n) for n in (na, nb, na + nb))
    a.upload(synth.operand(na, 1))
    b.upload(synth.operand(nb, 2))
    engine.launch_log(True)
    try:
        engine.mul_device(c.ptr, a.ptr, na, b.ptr, nb)
        cudart.synchronize()
        return [r[0] for r in engine.launch_records()]
    finally:
        engine.launch_log(False)
        for x in (a, b, c):
            x.free()


def test_these_primes_run(engine):
    # last in the module: what the tests above ran on. The 31-bit primes take
    # a short product in one launch, and all primes of a pass in one; here
    # each prime has launches of its own.
    assert engine.prime_set() == 2
    kinds = _launches(engine, 300, 200)
    assert "block_product" not in kinds and kinds.count("garner_carry") == 1, kinds
    passes = len(engine.plan(20))
    kinds = _launches(engine, 1 << 19, 1 << 19)
    assert kinds.count("fused_inner_pass") == 2 and kinds.count("fwd_pass_first") == 4, kinds
    assert kinds.count("fwd_pass") == 4 * (passes - 2), kinds
