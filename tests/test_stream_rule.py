"""Which products of 17 to 128 tokens the weight-streaming kernel takes: not those where the library's was measured ahead."""
import pytest


@pytest.mark.parametrize("m,n,k,gated,taken", [
    # heads: up to 96 tokens, not over a short K
    (96, 151936, 4096, False, True), (97, 151936, 4096, False, False), (128, 76000, 2048, False, False), (96, 151936, 1024, False, True),
    (128, 151936, 1024, False, False), (17, 76000, 512, False, False),
    # gate/up: beyond 96 tokens only wide ones, none beyond 112
    (96, 11264, 4096, True, True), (97, 11264, 4096, True, False), (112, 5632, 4096, True, False), (112, 24576, 4096, True, True),
    (113, 24576, 4096, True, False), (48, 16384, 2048, True, False), (32, 16384, 2048, True, True),
    # others: beyond 64 tokens only a long K and not too many rows
    (96, 28672, 8192, False, False), (96, 4096, 12288, False, True), (97, 4096, 12288, False, False), (65, 6144, 4096, False, False),
    (64, 6144, 4096, False, True), (32, 8192, 2048, False, True), (33, 8192, 2048, False, False), (17, 1024, 1024, False, False)])
def test_products_that_the_kernel_takes(m, n, k, gated, taken):
    from pulsar_b200 import ops
    assert ops._stream_wanted(m, n, k, gated) is taken
