"""Onesweep radix sort (sd_sort_pairs) against a stable CPU sort: bit-exact
keys and values for every key width, duplicate-heavy and ragged inputs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def run_sort(sd, keys, vals, key_bits):
    import torch
    n = len(keys)
    dev = torch.device("cuda:0")
    k = torch.from_numpy(keys.view(np.int32)).to(dev)
    v = torch.from_numpy(vals.view(np.int32)).to(dev)
    kt = torch.empty_like(k)
    vt = torch.empty_like(v)
    nb = sd.SpatialPartition.sort_scratch_bytes(n, key_bits)
    scratch = torch.zeros((nb + 3) // 4, dtype=torch.int32, device=dev)
    sd.SpatialPartition.sort_pairs(k, v, kt, vt, n, key_bits, scratch)
    assert sd.SpatialPartition.sort_status(scratch) == 0
    torch.cuda.synchronize()
    return k.cpu().numpy().view(np.uint32), v.cpu().numpy().view(np.uint32)


@pytest.mark.parametrize("n", [1, 2, 31, 2047, 2048, 2049, 100_000, 1_000_003])
@pytest.mark.parametrize("key_bits", [18, 20, 32])
def test_sort_random(sdlib, n, key_bits):
    rng = np.random.default_rng(n + key_bits)
    keys = rng.integers(0, 1 << key_bits, n, dtype=np.uint64).astype(np.uint32)
    vals = np.arange(n, dtype=np.uint32)
    k, v = run_sort(sdlib, keys, vals, key_bits)
    order = np.argsort(keys, kind="stable")
    assert np.array_equal(k, keys[order])
    assert np.array_equal(v, vals[order])


@pytest.mark.parametrize("key_bits", [1, 5, 8, 9, 10, 17, 19, 20, 21, 25, 27])
def test_sort_key_widths(sdlib, key_bits):
    rng = np.random.default_rng(key_bits)
    n = 300_000
    keys = rng.integers(0, 1 << key_bits, n, dtype=np.uint64).astype(np.uint32)
    vals = rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32)
    k, v = run_sort(sdlib, keys, vals, key_bits)
    order = np.argsort(keys, kind="stable")
    assert np.array_equal(k, keys[order]) and np.array_equal(v, vals[order])


@pytest.mark.parametrize("kind", ["all_equal", "two_values", "sorted", "reversed", "max_values", "few_runs"])
def test_sort_adversarial(sdlib, kind):
    n = 500_000
    rng = np.random.default_rng(1)
    if kind == "all_equal":
        keys = np.full(n, 12345, np.uint32)
    elif kind == "two_values":
        keys = rng.integers(0, 2, n).astype(np.uint32) * np.uint32(0xFFFF0000)
    elif kind == "sorted":
        keys = np.sort(rng.integers(0, 1 << 32, n, dtype=np.uint64)).astype(np.uint32)
    elif kind == "reversed":
        keys = np.sort(rng.integers(0, 1 << 32, n, dtype=np.uint64))[::-1].astype(np.uint32)
    elif kind == "max_values":
        keys = np.full(n, 0xFFFFFFFF, np.uint32)
        keys[::7] = 0
    else:
        keys = np.repeat(rng.integers(0, 1 << 32, 50, dtype=np.uint64).astype(np.uint32), n // 50)
    vals = np.arange(len(keys), dtype=np.uint32)
    k, v = run_sort(sdlib, keys, vals, 32)
    order = np.argsort(keys, kind="stable")
    assert np.array_equal(k, keys[order]) and np.array_equal(v, vals[order])


def test_sort_matches_oracle_on_hash_entries(sdlib, orc):
    """9n reference-layout entries of 200k spheres (1.8M pairs) sorted by the
    full cell word: identical to the oracle's stable LSD sort."""
    rng = np.random.default_rng(3)
    n = 200_000
    pos = np.zeros((n, 4), np.float32)
    pos[:, :3] = rng.uniform(0, 1, (n, 3))
    sizes = np.full(n, 0.004, np.float32)
    cells, spheres, count = orc.ref_hash_build(pos, sizes, 1.0 / 128)
    k, v = run_sort(sdlib, cells, spheres, 32)
    ko, vo = orc.radix_sort_pairs(cells, spheres, 32)
    assert np.array_equal(k, ko) and np.array_equal(v, vo)


def test_sort_empty_and_bad_args(sdlib):
    import ctypes as C
    import torch
    st = sdlib.lib().sd_sort_pairs(None, None, None, None, 0, 32, None, 0, None)
    assert st == 0
    x = torch.zeros(16, dtype=torch.int32, device="cuda")
    st = sdlib.lib().sd_sort_pairs(C.c_void_p(x.data_ptr()), C.c_void_p(x.data_ptr()), C.c_void_p(x.data_ptr()),
                                   C.c_void_p(x.data_ptr()), 16, 32, C.c_void_p(x.data_ptr()), 64, None)
    assert st == sdlib._abi.SD_ERR_CAPACITY  # scratch too small
    st = sdlib.lib().sd_sort_pairs(None, None, None, None, 16, 33, None, 0, None)
    assert st == sdlib._abi.SD_ERR_INVALID_ARG


@pytest.mark.parametrize("items", [8, 16])
@pytest.mark.parametrize("n", [32 * 4096 - 1, 32 * 4096, 32 * 4096 + 1, 33 * 4096, 64 * 4096 + 17, 700 * 2048 + 5])
@pytest.mark.parametrize("kind", ["random", "padded"])
def test_sort_look_back_groups(sdlib, items, n, kind):
    """Sizes around the look-back's groups of 32 tiles (2,048 or 4,096 keys),
    digits of 8, 9 and 10 bits, random keys and runs of one padding word, and
    key buffers off 16-byte alignment."""
    import torch
    rng = np.random.default_rng(n)
    before = sdlib._abi.tune_get("sort_items")
    sdlib._abi.tune_set("sort_items", items)
    try:
        for bits in (8, 18, 20, 32):
            keys = rng.integers(0, 1 << bits, n, dtype=np.uint64).astype(np.uint32)
            if kind == "padded":
                keys[rng.random(n) < 0.75] = (1 << bits) - 1
            dev = torch.device("cuda:0")
            buf = [torch.zeros(n + 1, dtype=torch.int32, device=dev)[1:] for _ in range(4)]
            buf[0].copy_(torch.from_numpy(keys.view(np.int32)))
            buf[1].copy_(torch.arange(n, dtype=torch.int32))
            scratch = torch.zeros(sdlib.SpatialPartition.sort_scratch_bytes(n, bits), dtype=torch.uint8, device=dev)
            sdlib.SpatialPartition.sort_pairs(*buf, n, bits, scratch)
            assert sdlib.SpatialPartition.sort_status(scratch) == 0
            order = np.argsort(keys, kind="stable")
            assert np.array_equal(buf[1].cpu().numpy(), order.astype(np.int32))
            assert np.array_equal(buf[0].cpu().numpy().view(np.uint32), keys[order])
    finally:
        sdlib._abi.tune_set("sort_items", before)


@pytest.mark.parametrize("n", [1, 4097, 300_000])
def test_chained_launches_in_streams_and_graphs(sdlib, orc, n):
    """Operators back to back on one stream, each on what the last one wrote,
    with the caller's own kernels and copies between them; and the same chain
    captured and replayed, where the launches are plain ones."""
    import torch
    P = sdlib.SpatialPartition
    rng = np.random.default_rng(n)
    host = rng.integers(0, 2 ** 32, n, dtype=np.uint32)
    src = torch.from_numpy(host.view(np.int32)).cuda()
    k, v, kt, vt = (torch.empty_like(src) for _ in range(4))
    scratch = torch.zeros((P.sort_scratch_bytes(n, 32) + 3) // 4, dtype=torch.int32, device="cuda")
    ids = torch.arange(n, dtype=torch.int32, device="cuda")

    def chain():
        k.copy_(src)
        v.copy_(ids)
        for _ in range(3):
            P.sort_collision_list(k, v, kt, vt, n, scratch)
            k.bitwise_not_()
        P.sort_collision_list(k, v, kt, vt, n, scratch)

    want_k, want_v = host, np.arange(n, dtype=np.uint32)
    for _ in range(3):
        want_k, want_v = orc.radix_sort_pairs(want_k, want_v, 32)
        want_k = ~want_k
    want_k, want_v = orc.radix_sort_pairs(want_k, want_v, 32)

    def check():
        torch.cuda.synchronize()
        assert np.array_equal(k.cpu().numpy().view(np.uint32), want_k)
        assert np.array_equal(v.cpu().numpy().view(np.uint32), want_v)

    chain()
    check()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(4):
            chain()
    check()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        chain()
    for t in (k, v, kt, vt):
        t.zero_()
    for _ in range(3):
        graph.replay()
    check()
