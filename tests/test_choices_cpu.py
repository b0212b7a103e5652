"""Host-side choices that shape launches (no GPU): the length bucket and the number of key splits."""
from trapetum_b200.csrc.ops import choose_decode_splits
from trapetum_b200.engine import len_bucket


def test_len_bucket_is_a_power_of_two_not_below():
    assert len_bucket(1) == 256 and len_bucket(256) == 256 and len_bucket(257) == 512
    assert len_bucket(8192) == 8192 and len_bucket(8193) == 16384
    for n in (3, 100, 1000, 5000):
        b = len_bucket(n)
        assert b >= n and b & (b - 1) == 0


def test_decode_splits():
    # one sequence: many pieces, to put a CTA on as many SMs as the pages allow (at least 4 pages each)
    assert choose_decode_splits(1, 4, 128, 148) == 31
    # a short context is not cut
    assert choose_decode_splits(8, 4, 4, 148) == 1 and choose_decode_splits(1, 4, 7, 148) == 1
    # 32 (sequence, kv head) pairs on 148 SMs: four pieces fill one round
    assert choose_decode_splits(8, 4, 128, 148) == 4
    # 256 pairs: one piece would leave most of a second round idle
    assert choose_decode_splits(64, 4, 128, 148) == 4
    for batch in (1, 3, 8, 64, 200):
        for pages in (1, 9, 64, 128, 1000):
            s = choose_decode_splits(batch, 4, pages, 148)
            assert 1 <= s <= 64 and (s == 1 or pages // s >= 4)


def test_unevenness_and_the_partition_it_chooses():
    """The engine tells the kernels how much a batch's contexts differ (in quarters of batch x longest that are
    empty); it is part of the key of a captured decode step.  Decode attention deals its pages out as one stream
    only where that saves more than a streaming launch costs."""
    from trapetum_b200.csrc.ops import decode_partition_is_stream
    from trapetum_b200.engine.engine import uneven_lengths, unevenness
    assert unevenness([8000]) == 0                          # one sequence is never uneven
    assert unevenness([8000, 8000, 7000, 8192]) == 0
    assert unevenness([3, 3, 4]) == 0
    assert unevenness([4, 4, 4, 4]) == 0 and unevenness([4, 4, 4, 0]) == 0 and unevenness([4, 4, 3, 0]) == 1
    assert unevenness([8, 8, 0, 0]) == 1 and unevenness([8, 7, 0, 0]) == 2 and unevenness([8, 0, 0, 0]) == 2
    assert unevenness([8, 0, 0, 0, 0]) == 3
    assert unevenness([8000, 100, 100, 100]) == 2 and unevenness([8000] + [64] * 7) == 3
    assert unevenness([1, 1, 1, 64]) == 2
    assert uneven_lengths([8000, 100, 100, 100]) and not uneven_lengths([5, 5])
    # prompts of 64 to 2,048 tokens in a batch of 8 (sum 8,305 of 8 x 1,919), 9B heads: pieces of 16 pages, a
    # quarter of which a stream would save: the sequences are cut
    lens = [1555, 532, 1206, 836, 1919, 144, 1149, 964]
    assert unevenness(lens) == 1
    assert not decode_partition_is_stream(8, 8, 32, choose_decode_splits(8, 8, 32, 148), 1, 148)
    # one long sequence among short ones: 32-page pieces, three quarters saved: one stream
    assert decode_partition_is_stream(8, 4, 128, choose_decode_splits(8, 4, 128, 148), 3, 148)
    # equal lengths: a stream only where the pieces would take more than two rounds of CTAs
    assert not decode_partition_is_stream(8, 4, 128, 4, 0, 148) and not decode_partition_is_stream(64, 4, 32, 1, 0, 148)
    assert decode_partition_is_stream(64, 16, 32, 1, 0, 148)


def test_latent_decode_pieces_are_near_the_best_that_was_timed():
    """(sequences, heads, bucket of rows) and us a launch by the number of pieces, timed on a B200 at three quarters of
    the bucket: the chosen number takes at most a sixth more than the best one."""
    import ctypes

    from trapetum_b200.csrc import build
    pieces = build.load("attention_latent").tb_latent_decode_pieces
    timed = {(1, 16, 512): {1: 22.2, 2: 17.0, 3: 16.2, 4: 13.7, 5: 16.2, 6: 16.4},
             (1, 16, 4096): {8: 21.3, 12: 19.9, 16: 20.0, 18: 20.3, 24: 19.3, 32: 19.6, 40: 21.5, 48: 23.2, 64: 26.1},
             (2, 32, 4096): {4: 30.8, 8: 21.5, 12: 20.2, 18: 20.8, 24: 19.6, 28: 20.2, 32: 21.4, 40: 24.6, 48: 33.1},
             (3, 16, 2048): {4: 20.9, 6: 20.6, 7: 19.0, 8: 16.4, 9: 19.3, 12: 17.3, 16: 18.5, 20: 19.2, 24: 18.9},
             (3, 32, 4096): {4: 31.6, 8: 21.3, 12: 20.4, 16: 20.4, 18: 21.3, 20: 21.1, 24: 28.6, 28: 25.9, 32: 31.4},
             (5, 16, 4096): {4: 31.9, 8: 21.3, 12: 20.4, 16: 22.3, 18: 22.4, 20: 22.4, 24: 22.3, 28: 23.9, 32: 31.9},
             (6, 16, 4096): {4: 31.7, 8: 21.3, 12: 21.6, 16: 22.5, 18: 22.5, 20: 22.4, 24: 28.0, 28: 25.9, 32: 32.3},
             (8, 16, 4096): {4: 31.8, 7: 27.2, 8: 21.4, 9: 25.0, 12: 21.8, 16: 24.0, 18: 26.9, 20: 24.9, 24: 33.7},
             (5, 32, 2048): {4: 21.9, 7: 19.2, 8: 18.8, 9: 19.7, 10: 20.0, 12: 20.4, 14: 23.8, 16: 28.1, 20: 28.4},
             (12, 16, 2048): {4: 24.8, 6: 24.4, 7: 21.8, 8: 21.0, 9: 21.3, 10: 21.7, 12: 23.6, 14: 31.9, 20: 34.3},
             (20, 16, 4096): {2: 65.3, 3: 49.9, 4: 39.1, 6: 33.3, 7: 31.5, 8: 46.5, 12: 42.4, 20: 51.5},
             (48, 16, 4096): {1: 92.4, 2: 53.2, 3: 44.9, 4: 62.8, 6: 54.3, 8: 66.5},
             (64, 16, 4096): {1: 120.0, 2: 67.9, 3: 91.4, 4: 78.6, 6: 87.5, 8: 98.3}}
    for (batch, heads, rows), us in timed.items():
        n = pieces(*map(ctypes.c_int, (batch, heads, rows, 148)))
        at = us[min(us, key=lambda k: abs(k - n))]
        assert at <= min(us.values()) * 7 / 6, (batch, heads, rows, n)
    for batch in (1, 3, 16, 64, 200, 1000):                        # and any call gets at least one piece of a tile or more
        for rows in (1, 32, 100, 5000, 1 << 20):
            n = pieces(*map(ctypes.c_int, (batch, 16, rows, 148)))
            assert 1 <= n <= 64 and (n == 1 or n * 32 <= rows)


def test_every_way_of_cutting_latent_rows_has_a_test():
    """The sizes of the GPU tests of decode attention over cached latents reach one, two, four and eight pieces that meet in a
    cluster, and more that a launch folds."""
    import ctypes

    import test_gpu_kernels as gpu
    from trapetum_b200.csrc import build
    lib = build.load("attention_latent")
    cases = [(c[0], c[1], min(c[4], c[5] + 31) if c[5] else c[4]) for c in gpu.LATENT_CLUSTERS + gpu.LATENT_FOLDED]
    seen = set()
    for i, (batch, heads, rows) in enumerate(cases):
        n = lib.tb_latent_decode_pieces(*map(ctypes.c_int, (batch, heads, rows, 148)))
        folds = bool(lib.tb_latent_decode_folds(*map(ctypes.c_int, (n, batch, heads))))
        assert folds == (i >= len(gpu.LATENT_CLUSTERS))
        seen.add("folds" if folds else n)
    assert seen == {1, 2, 4, 8, "folds"}


def test_the_gated_norm_of_few_tokens_uses_the_threads_there_are():
    """A step of few tokens is a chain of waits: 1,024 threads a row, one group of four columns each as long as that goes."""
    import ctypes

    from trapetum_b200.csrc import build
    groups = build.load("mamba2").tb_mamba2_gate_norm_groups
    for tokens, threads in ((1, 1024), (64, 1024), (65, 256), (2048, 256)):
        for gs in (4, 1000, 1024, 4096, 4100, 8192, 16384):
            n = groups(ctypes.c_int(tokens), ctypes.c_int(gs))
            assert n in (1, 2, 4, 8, 16) and gs <= 4 * threads * n and (n == 1 or gs > 2 * threads * n)
