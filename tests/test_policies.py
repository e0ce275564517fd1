"""Host-side choices that need no GPU: how many blocks the decode attention gives a (token, KV head)
pair, and how many K slices a decode-sized product is cut into."""
import numpy as np

from inferllm_b200.kernels import ops


def test_decode_attention_splits_stay_in_range_and_follow_the_measurements():
    for pairs in (1, 8, 32, 64, 96, 128, 160, 192, 256, 320, 384, 512, 1280, 2048):
        for ctx in (1, 64, 65, 512, 1024, 4096, 32768):
            n = ops.attention_decode_ring_splits(pairs, 1, ctx)
            tiles = -(-ctx // 64)
            assert 1 <= n <= min(tiles, 32), (pairs, ctx, n)
    # a grid a little larger than the 296 blocks that run at once is cut into several waves
    # (measured: 320 pairs at context 4096, 129 us in one split, 106 us in six)
    assert 4 <= ops.attention_decode_ring_splits(8, 40, 4096) <= 8
    # grids that fill the GPU in one wave, or in many, stay whole (160 pairs: 56 us in one split,
    # 69 us in two; 512 pairs at context 1024: 44 us in one split, 50 us in two)
    assert ops.attention_decode_ring_splits(5, 32, 4096) == 1
    assert ops.attention_decode_ring_splits(8, 32, 4096) == 1
    assert ops.attention_decode_ring_splits(16, 32, 1024) == 1
    assert ops.attention_decode_ring_splits(64, 32, 4096) == 1
    # few pairs are split until about 160 blocks are at work, never into more blocks than tiles
    assert ops.attention_decode_ring_splits(1, 8, 32768) >= 16
    assert ops.attention_decode_ring_splits(1, 32, 64) == 1
    # the head size scales the bytes a block streams and with them what a split is worth
    assert ops.attention_decode_ring_splits(8, 8, 4096, 64) <= ops.attention_decode_ring_splits(8, 8, 4096, 128) + 1


def test_split_k_of_decode_sized_products():
    for M in (1, 8, 16, 64):
        for N, K in ((4096, 4096), (12288, 4096), (22016, 4096), (4096, 11008), (32000, 4096), (100, 64), (128, 8)):
            n = ops.gemm_tc_splits(M, N, K)
            k_iters = -(-K // 64)
            assert 1 <= n <= 8 and n <= k_iters
            per = -(-k_iters // n)
            assert per * (n - 1) < k_iters          # every slice owns at least one 64-wide piece of K
    assert ops.gemm_tc_splits(65, 4096, 4096) == 1   # larger steps are not split
    assert ops.gemm_tc_splits(8, 22016, 4096) == 1   # 172 tiles fill the GPU by themselves
    assert ops.gemm_tc_splits(8, 4096, 4096) == 8


def test_how_generic_attention_takes_a_steps_tokens():
    """Tokens by eights where the tiles of one or two sequences fill the SMs, single tokens beside them one by one; the counts against a
    walk over the tokens."""
    form = lambda lens, heads=32: ops.attention_generic_form(lens, heads, 148)  # noqa: E731
    rng = np.random.default_rng(0)
    for _ in range(300):
        lens = rng.choice([0, 1, 2, 3, 7, 8, 9, 17, 40], rng.integers(1, 12)).tolist()
        seqs = np.repeat(np.arange(len(lens)), lens)
        tiles = [seqs[i:i + 8] for i in range(0, len(seqs), 8)]
        dense = sum(3 * len(set(t.tolist())) <= len(t) for t in tiles)
        assert form(lens)[1:] == (dense, len(tiles) - dense), lens
    assert form([512]) == (1, 64, 0) and form([300, 200, 100])[0] == 1 and form([20] * 8)[0] == 1
    assert form([512] + [1] * 40) == (2, 64, 5)         # the single tokens' tiles are not walked by eights
    assert form([1] * 64)[0] == 0 and form([17] + [1] * 63)[0] == 0 and form([3] * 4)[0] == 0
    assert form([64], heads=4)[0] == 0 and form([17], heads=4)[0] == 0      # few blocks: a block per token


def test_differential_decode_splits():
    """At most one block per 256 keys of the longest sequence and at most 64; about two blocks per SM in all; one for
    steps of many tokens; the same for every step of a shape (it looks at the cache's limit, not at the sequences)."""
    for pairs in (1, 8, 16, 64, 256, 1024, 4096):
        for longest in (1, 256, 257, 4096, 131072):
            n = ops.attention_diff_splits(pairs, 1, longest, 148)
            assert 1 <= n <= min(-(-longest // 256), 64), (pairs, longest, n)
            assert n == 1 or pairs * n <= 2 * 148
    assert ops.attention_diff_splits(8, 8, 4096, 148) == 4
    assert ops.attention_diff_splits(8, 2, 4096, 148) == 16
    assert ops.attention_diff_splits(512, 8, 4096, 148) == 1


def test_who_takes_a_recurrences_tokens():
    """Chunks of eight where they were measured to be the faster ones, the older kernels elsewhere, in the bfloat16 mode (1, 0 and 2: ops.scan_form)."""
    linear, channel, head = (lambda *a, k=k: ops.scan_form(k, *a) for k in (0, 1, 2))
    for form in (linear, channel, head):        # T, B, longest, heads, key and value channels
        assert form(8, 1, 8, 16, 128, 128) == 0 and form(480, 32, 15, 16, 128, 128) == 0
        assert form(4096, 4, 1500, 16, 128, 128) == 1
    assert [channel(4096, 1, 4096, 16, d, 128) for d in (16, 48, 64, 128, 129, 256)] == [0, 1, 1, 1, 0, 0]
    assert [head(4096, 4, 1500, 16, d, 128) for d in (16, 48, 64, 128, 129, 256)] == [2, 2, 2, 1, 2, 2]
    assert channel(48, 1, 48, 16, 128, 128) == 0 and channel(48, 1, 48, 32, 128, 128) == 1 and channel(600, 1, 600, 2, 64, 64) == 1
    assert channel(6254, 32, 300, 32, 64, 128) == 0 and channel(6254, 32, 300, 32, 128, 128) == 1
    assert head(16, 1, 16, 32, 128, 128) == 0 and head(600, 1, 600, 2, 128, 128) == 2 and head(2334, 32, 100, 16, 128, 128) == 1 and head(2334, 32, 100, 16, 64, 64) == 0
    assert linear(2048, 1, 2048, 2, 32, 32) == 1 and linear(2048, 1, 2048, 16, 129, 128) == 0
    assert linear(346, 32, 16, 8, 128, 128) == 0 and linear(41, 4, 16, 8, 128, 128) == 1 and linear(60, 1, 60, 8, 64, 64) == 1 and linear(172, 8, 32, 32, 32, 64) == 0
    assert linear(8353, 32, 400, 32, 32, 256) == 0 and linear(8353, 32, 400, 32, 64, 128) == 0 and linear(8353, 32, 400, 32, 128, 128) == 1
