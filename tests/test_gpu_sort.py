"""GPU radix sort: equals a stable sort by the low `bits` of each key (sm_100a)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 100, 4095, 4096, 4097, 6143, 6144, 6145, 100000, 1 << 20])
@pytest.mark.parametrize("kb,bits", [(4, 32), (4, 30), (4, 13), (8, 60), (8, 64), (8, 41)])
def test_radix_sort_stable(ctx, n, kb, bits):
    rng = np.random.default_rng(n * 131 + bits)
    if kb == 4:
        keys = rng.integers(0, 1 << 32, size=n, dtype=np.uint64).astype(np.uint32)
        keys[: n // 3] = keys[0]  # a long run of duplicates
        K = torch.from_numpy(keys.view(np.int32)).cuda()
        mask = np.uint32((1 << bits) - 1) if bits < 32 else np.uint32(0xffffffff)
        sk = keys & mask
    else:
        keys = rng.integers(0, 1 << 63, size=n, dtype=np.uint64) * np.uint64(2) + rng.integers(0, 2, size=n,
                                                                                             dtype=np.uint64)
        keys[: n // 3] = keys[0]
        K = torch.from_numpy(keys.view(np.int64)).cuda()
        mask = np.uint64((1 << bits) - 1) if bits < 64 else np.uint64(0xffffffffffffffff)
        sk = keys & mask
    ko, vo = ctx.radix_sort(K, bits=bits)
    ctx.check()
    order = np.argsort(sk, kind="stable")
    np.testing.assert_array_equal(vo.cpu().numpy(), order.astype(np.int32))
    got = ko.cpu().numpy().view(keys.dtype)
    np.testing.assert_array_equal(got, keys[order])


def test_radix_sort_with_values(ctx):
    rng = np.random.default_rng(1)
    keys = rng.integers(0, 1 << 20, size=300000).astype(np.uint32)
    vals = rng.integers(-5, 5, size=300000).astype(np.int32)
    ko, vo = ctx.radix_sort(torch.from_numpy(keys.view(np.int32)).cuda(), torch.from_numpy(vals).cuda(), bits=20)
    order = np.argsort(keys, kind="stable")
    np.testing.assert_array_equal(vo.cpu().numpy(), vals[order])


def _wide_case(kind, n, bits, rng):
    """Keys for the wide-key path (bits > 48): the array is first ordered by its top
    24 sorted bits, then every run of equal top bits is sorted by the rest, in
    shared memory, or by the large-segment kernel when a run exceeds 2,048 keys.
    The top 16 bits are chosen here, so a run has about 1/256 of a prefix's keys."""
    low = rng.integers(0, 1 << (bits - 16), size=n, dtype=np.uint64)
    if kind == "uniform":
        top = rng.integers(0, 1 << 16, size=n, dtype=np.uint64)
    elif kind == "skewed":
        # one prefix with 30 % of the keys, 40 prefixes of 3,000-6,000 keys
        # around the shared-memory capacity, the rest spread out
        top = rng.integers(0, 1 << 16, size=n, dtype=np.uint64)
        top[: int(0.3 * n)] = 777
        sizes = rng.integers(3000, 6000, size=40)
        pos = int(0.3 * n)
        for k, m in enumerate(sizes):
            top[pos:pos + m] = 1000 + k
            pos += m
        rng.shuffle(top)
    else:  # one prefix only
        top = np.full(n, 4242, np.uint64)
    keys = (top << np.uint64(bits - 16)) | low
    keys[: n // 50] = keys[0]  # duplicates
    if bits < 64:  # bits above the sorted width are carried, not sorted
        keys |= rng.integers(0, 2, size=n, dtype=np.uint64) << np.uint64(63)
    return keys


@pytest.mark.parametrize("kind,n,bits", [("uniform", (1 << 20) + 123, 60), ("uniform", 3 << 20, 64),
                                         ("uniform", 1 << 21, 49), ("skewed", 1 << 21, 60),
                                         ("skewed", (1 << 20) + 7, 56), ("single", 1 << 20, 60)])
@pytest.mark.parametrize("with_vals", [False, True])
def test_radix_sort_wide_keys_by_segments(ctx, kind, n, bits, with_vals):
    rng = np.random.default_rng(n + bits + (7 if with_vals else 0))
    keys = _wide_case(kind, n, bits, rng)
    mask = np.uint64((1 << bits) - 1) if bits < 64 else np.uint64(0xffffffffffffffff)
    K = torch.from_numpy(keys.view(np.int64)).cuda()
    vals = rng.permutation(n).astype(np.int32) if with_vals else None
    ko, vo = ctx.radix_sort(K, None if vals is None else torch.from_numpy(vals).cuda(), bits=bits)
    ctx.check()
    order = np.argsort(keys & mask, kind="stable")
    np.testing.assert_array_equal(vo.cpu().numpy(), (vals[order] if with_vals else order.astype(np.int32)))
    np.testing.assert_array_equal(ko.cpu().numpy().view(np.uint64), keys[order])


@pytest.mark.parametrize("dtype", [np.uint32, np.uint64])
@pytest.mark.parametrize("n", [31, 1023, 1024, 1025, 8191, 8192, 8193, 12289])
@pytest.mark.parametrize("kind", ["uniform", "few", "equal"])
def test_sort_one_cta_edges(ctx, dtype, n, kind):
    """Around the largest sort of one CTA (8,192 keys) and of its rounds of 1,024, for
    both key widths; wide keys go on with the segmented sort from there."""
    rng = np.random.default_rng(n)
    bits = 30 if dtype == np.uint32 else 60
    keys = {"uniform": rng.integers(0, 1 << bits, size=n, dtype=np.uint64),
            "few": rng.integers(0, 7, size=n, dtype=np.uint64) << np.uint64(bits - 9),
            "equal": np.full(n, 5, np.uint64)}[kind].astype(dtype)
    vals = rng.permutation(n).astype(np.int32)
    order = np.argsort(keys, kind="stable")
    K = torch.from_numpy(keys.view(np.int32 if dtype == np.uint32 else np.int64)).cuda()
    ko, vo = ctx.radix_sort(K, torch.from_numpy(vals).cuda(), bits=bits)
    ctx.check()
    np.testing.assert_array_equal(ko.cpu().numpy().view(dtype), keys[order])
    np.testing.assert_array_equal(vo.cpu().numpy(), vals[order])


def _long_case(kind, n, bits, rng):
    """Wide keys with runs of equal top 24 bits around the sizes where k_seg_big goes from
    a CTA per run to chunks (8,192 keys; a chunk of these arrays is 2,048 or, of the largest, 6,144)."""
    low = rng.integers(0, 1 << (bits - 24), size=n, dtype=np.uint64)
    if kind == "one":
        top = np.full(n, 9, np.uint64)
    elif kind == "outlier":
        top = np.zeros(n, np.uint64)
        top[n // 3] = (1 << 24) - 1
    else:  # whole runs, chunked ones and short ones together
        sizes, left = [], n
        for m in (8191, 8192, 8193, 2048, 2049, 10240, 10241, 5, 20000) * (n // 60000 + 1):
            sizes.append(min(m, left))
            left -= sizes[-1]
        sizes.append(left)
        top = np.repeat(np.arange(len(sizes), dtype=np.uint64) * np.uint64(3), sizes)
        top = top[rng.permutation(n)]
    low[: n // 50] = low[0]
    return (top << np.uint64(bits - 24)) | low


@pytest.mark.parametrize("kind", ["one", "outlier", "mixed"])
@pytest.mark.parametrize("n,bits,with_vals", [(8193, 60, False), (16385, 64, True), (100003, 60, True),
                                              (70001, 49, False), (131072, 56, True), (700001, 60, False)])
def test_radix_sort_long_runs(ctx, kind, n, bits, with_vals):
    rng = np.random.default_rng(n + len(kind))
    keys = _long_case(kind, n, bits, rng)
    vals = rng.permutation(n).astype(np.int32) if with_vals else None
    K = torch.from_numpy(keys.view(np.int64)).cuda()
    for block in (512, 256):
        ctx.set_tune(sort_block=block)
        try:
            ko, vo = ctx.radix_sort(K, None if vals is None else torch.from_numpy(vals).cuda(), bits=bits)
            ctx.check()
        finally:
            ctx.reset_tune()
        order = np.argsort(keys, kind="stable")
        np.testing.assert_array_equal(vo.cpu().numpy(), vals[order] if with_vals else order.astype(np.int32))
        np.testing.assert_array_equal(ko.cpu().numpy().view(np.uint64), keys[order])


@pytest.mark.parametrize("n", [100003, 1048573])
def test_one_prefix_costs_little_more(ctx, n):
    """Keys under one prefix take no more than four times as long as spread ones (twice, as
    measured; 19 and 120 times when one CTA sorted them)."""
    rng = np.random.default_rng(n)
    low = rng.integers(0, 1 << 36, size=n, dtype=np.uint64)
    ms = {}
    for kind, top in (("spread", rng.integers(0, 1 << 24, size=n, dtype=np.uint64)), ("one", np.full(n, 9, np.uint64))):
        K = torch.from_numpy(((top << np.uint64(36)) | low).view(np.int64)).cuda()
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        got = []
        for _ in range(9):
            a.record()
            ctx.radix_sort(K, bits=60)
            b.record()
            b.synchronize()
            got.append(a.elapsed_time(b))
        ms[kind] = sorted(got)[4]
    ctx.check()
    assert ms["one"] < 4 * ms["spread"], ms
