"""The host-side plans of the kernel library (no GPU): how keys are cut into slices and K into splits."""
import pytest

from safetyraise_lmengine_b200.kernels.library import KernelLibrary


@pytest.mark.parametrize("n_entries", [1, 2, 3, 8, 17, 64, 300])
@pytest.mark.parametrize("nkv", [1, 2, 8])
@pytest.mark.parametrize("max_kv", [1, 63, 64, 65, 2083, 8192, 40000])
@pytest.mark.parametrize("cap", [8, 32])
def test_attention_split_covers_every_key_in_whole_tiles(n_entries, nkv, max_kv, cap):
    nsplit, chunk = KernelLibrary.attention_split(n_entries, nkv, max_kv, max_slices=cap)
    assert 1 <= nsplit <= cap
    assert chunk > 0 and chunk % 64 == 0
    assert nsplit * chunk >= max_kv                       # every key lies in a slice
    assert (nsplit - 1) * chunk < max(max_kv, 1) + 63     # and no slice is empty
    # within one wave of two blocks per SM, unless a single slice per pair is already more
    assert nsplit == 1 or n_entries * nkv * nsplit <= 296


@pytest.mark.parametrize("M", [1, 8, 9, 16, 17, 32, 33, 64, 65, 128, 129, 300, 512, 1024, 2048, 5000])
@pytest.mark.parametrize("N, K", [(6144, 4096), (4096, 4096), (24576, 4096), (4096, 12288), (151936, 4096),
                                  (200, 72), (128, 64), (1024, 25600)])
def test_gemm_splits_keeps_its_bounds(M, N, K):
    sp = KernelLibrary.gemm_splits(M, N, K)
    total_kb = (K + 63) // 64
    assert 1 <= sp <= max(1, total_kb)
    if sp > 1:
        assert total_kb // sp >= 4                        # a split keeps at least a few k-blocks
    bn = KernelLibrary.gemm_token_tile(M, N)
    if bn == 256:
        assert sp == 1                                    # pairs of SMs on whole tiles of 256 x 256
    assert KernelLibrary.gemm_token_tile(512, 5120) == 256 and KernelLibrary.gemm_token_tile(512, 4096) == 128
    assert KernelLibrary.gemm_token_tile(2048, 4096) == 256 and KernelLibrary.gemm_token_tile(300, 5120) == 128
    if sp > 8:                                            # beyond a cluster: the partial sums fit the workspace
        tiles = ((N + 127) // 128) * ((M + bn - 1) // bn)
        assert 65536 + sp * tiles * 128 * bn * 4 <= KernelLibrary.GEMM_WS_BYTES


# us of the dense product with its activation in tiles of 256 and of 128 tokens, as measured
@pytest.mark.parametrize("tokens, features, us_256, us_128", [
    (256, 4096, 17.3, 13.0), (500, 4096, 18.2, 14.0), (640, 4096, 17.9, 18.9), (2048, 4096, 28.1, 32.9),
    (256, 8192, 23.3, 19.1), (300, 8192, 24.1, 29.0), (640, 8192, 35.6, 40.0), (256, 12288, 31.1, 39.6), (300, 12288, 46.2, 40.5),
    (384, 12288, 46.7, 40.8), (500, 12288, 48.0, 57.5), (256, 16384, 39.3, 51.6), (300, 16384, 57.7, 70.8), (300, 20480, 92.3, 107.8)])
def test_dense_tiles_are_the_faster_ones(tokens, features, us_256, us_128):
    from safetyraise_lmengine_b200.kernels import ops
    assert ops.dense_tile_rows(tokens, features) == (256 if us_256 < us_128 else 128)


def test_prefill_attention_plan():
    plan = KernelLibrary.prefill_attention_plan
    # a whole prompt of 2,048 tokens, 4 heads per KV head, 8 KV heads: enough blocks of two row tiles, no slices
    assert plan([8192], [2048], 8, 148) == (2, 1, 0)
    # a portion of 512 tokens behind 30,000: 64 blocks of two row tiles; the keys go in slices of whole tiles
    tiles, nsplit, chunk = plan([2048], [30512], 8, 148)
    assert tiles == 2 and nsplit >= 2 and chunk % 128 == 0 and nsplit * chunk >= 30512 > (nsplit - 1) * chunk
    # 152 lone row tiles would need two rounds of the GPU, 80 blocks of two tiles one: two tiles, no slices
    assert plan([2405], [1505], 8, 148) == (2, 1, 0)
    # a handful of rows and keys: nothing to cut
    assert plan([5], [100], 1, 148)[1:] == (1, 0)
    for rows, kv, nkv in (([1, 4000], [9000, 4000], 2), ([300] * 40, [5000] * 40, 8), ([128], [257], 1)):
        tiles, nsplit, chunk = plan(rows, kv, nkv, 148)
        assert tiles in (1, 2) and 1 <= nsplit <= 16
        if nsplit > 1:
            assert tiles == 2 and chunk % 128 == 0 and nsplit * chunk >= max(kv) > (nsplit - 1) * chunk - 128


def test_native_uniform_numbers_are_those_of_the_plain_function():
    import random

    import numpy as np
    import pytest
    from safetyraise_lmengine_b200.sampling.sampler import fill_uniforms, uniform_for
    r = random.Random(5)
    seeds = [r.randrange(-9, 1 << 64) for _ in range(300)] + [0, -1, (1 << 64) - 1]
    indices = [r.randrange(1 << 31) for _ in seeds]
    out = np.empty(len(seeds), dtype=np.float32)
    fill_uniforms(seeds, indices, out)
    assert out.tolist() == [uniform_for(s, i) for s, i in zip(seeds, indices)]
    for args in ((seeds, indices, out[1:]), (seeds[1:], indices, out[1:]), (seeds[2:], indices, out[1:])):
        with pytest.raises(ValueError):
            fill_uniforms(*args)
