"""Which log-probabilities one launch reads off: those where it is faster than the library's sort."""
import pytest


@pytest.mark.parametrize("V,k,ok", [(32000, 5, True), (32000, 64, True), (32000, 65, False), (128256, 20, True), (128256, 32, False),
                                    (256000, 10, True), (256000, 20, False), (256000, 0, True), (7, 7, True), (7, 8, False), (1000, -1, False)])
def test_rule(V, k, ok):
    from vllm_b200.ops.cuda import logprobs_ok
    assert logprobs_ok(V, k) is ok
