"""Sweep and prune on the GPU: the reference's windowed sweep rows against
the reference kernel's own output (tests/golden/ref_sap_*.npz) and the
oracle, and the exact pair operator against the oracle's pair sets."""
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
GOLDEN = Path(__file__).resolve().parent / "golden"


@pytest.mark.parametrize("case", ["a", "b"])
def test_sap_sweep_matches_reference_kernel(sdlib, case):
    import torch
    g = np.load(GOLDEN / f"ref_sap_{case}.npz")
    t = lambda k: torch.from_numpy(np.ascontiguousarray(g[k])).cuda()
    rows = sdlib.SweepAndPrune.sweep(t("upperx"), t("lowerx_sorted"), t("uppery"), t("lowery"), t("idx_sorted"))
    assert np.array_equal(rows.cpu().numpy(), g["rows"])
    rows2 = sdlib.SweepAndPrune.process_collisions(t("pos"))
    assert np.array_equal(rows2.cpu().numpy(), g["rows"])


@pytest.mark.parametrize("n,seed", [(0, 0), (1, 0), (2, 1), (5000, 2), (200_000, 3)])
def test_sap_process_matches_oracle(sdlib, orc, n, seed):
    import torch
    rng = np.random.default_rng(seed)
    pos = np.zeros((n, 4), np.float32)
    pos[:, :3] = rng.uniform(0.0, 1.0, (n, 3))
    pos[:, 3] = rng.uniform(0.001, 0.01, n)
    rows = sdlib.SweepAndPrune.process_collisions(torch.from_numpy(pos).cuda())
    assert np.array_equal(rows.cpu().numpy(), orc.sap_process(pos))


@pytest.mark.parametrize("n,seed", [(0, 0), (1, 0), (2, 1), (3000, 4), (100_000, 5)])
def test_sap_pairs_bit_exact(sdlib, orc, n, seed):
    import torch
    rng = np.random.default_rng(seed)
    c = rng.uniform(-0.4, 1.6, (n, 3)).astype(np.float32)
    h = rng.uniform(0.001, 0.015, (n, 3)).astype(np.float32)
    L = np.zeros((n, 4), np.float32)
    H = np.zeros((n, 4), np.float32)
    L[:, :3] = c - h
    H[:, :3] = c + h
    if n >= 2:
        L[1], H[1] = L[0], H[0]
    want = orc.aabb_pairs(L, H)
    got, cnt, err = sdlib.SweepAndPrune.pairs(torch.from_numpy(L).cuda(), torch.from_numpy(H).cuda(), len(want) + 8)
    assert err == 0 and cnt == len(want)
    assert np.array_equal(got.cpu().numpy().view(np.uint64), want)


def test_sap_pairs_overflow_is_reported(sdlib):
    import torch
    rng = np.random.default_rng(9)
    c = rng.uniform(0, 1, (2000, 3)).astype(np.float32)
    L = np.zeros((2000, 4), np.float32)
    H = np.zeros((2000, 4), np.float32)
    L[:, :3] = c - 0.05
    H[:, :3] = c + 0.05
    got, cnt, err = sdlib.SweepAndPrune.pairs(torch.from_numpy(L).cuda(), torch.from_numpy(H).cuda(), 10)
    assert err & sdlib._abi.SD_DEVERR_PAIR_OVERFLOW


def _scene(kind, n, seed):
    """Boxes that stress the binned sweep's column grid: mixed sizes with a
    few boxes spanning the domain, corners on column boundaries, a flat
    scene (no y-z extent at all), y/z-inverted boxes, large coordinates."""
    rng = np.random.default_rng(seed)
    c = rng.uniform(-0.7, 1.3, (n, 3)).astype(np.float32)
    h = np.exp(rng.normal(np.log(0.006), 0.6, (n, 3))).astype(np.float32)
    if kind == "mixed":
        h[rng.random(n) < 0.01] = 0.0
        big = rng.random(n) < 0.002
        h[big] = rng.uniform(0.2, 0.9, (int(big.sum()), 3))
    elif kind == "aligned":
        c = (rng.integers(0, 96, (n, 3)) / 64.0).astype(np.float32)
        h = (rng.integers(0, 3, (n, 3)) / 128.0).astype(np.float32)
    elif kind == "flat":
        c[:, 1:] = 0.5
        h[:, 1:] = 0.0
    elif kind == "large":
        c = (c * 1000.0 + 1.0e6).astype(np.float32)
        h = (h * 1000.0).astype(np.float32)
    L = np.zeros((n, 4), np.float32)
    H = np.zeros((n, 4), np.float32)
    L[:, :3] = c - h
    H[:, :3] = c + h
    if kind == "inverted_yz":
        flip = rng.random(n) < 0.1
        L[flip, 1], H[flip, 1] = H[flip, 1].copy(), L[flip, 1].copy()
        flip = rng.random(n) < 0.1
        L[flip, 2], H[flip, 2] = H[flip, 2].copy(), L[flip, 2].copy()
    return L, H


@pytest.mark.parametrize("kind", ["mixed", "aligned", "flat", "inverted_yz", "large"])
def test_sap_pairs_binned_edge_cases(sdlib, orc, kind):
    """The binned sweep (columns, one report per pair in the column of the
    overlap's lower y-z corner) finds exactly the oracle's pair set."""
    import torch
    L, H = _scene(kind, 20_000 if kind != "flat" else 4000, seed=len(kind))
    want = orc.aabb_pairs(L, H)
    got, cnt, err = sdlib.SweepAndPrune.pairs(torch.from_numpy(L).cuda(), torch.from_numpy(H).cuda(), len(want) + 8)
    assert err == 0 and cnt == len(want), (kind, cnt, len(want), err)
    assert np.array_equal(got.cpu().numpy().view(np.uint64), want)


@pytest.mark.parametrize("op", ["sap", "lbvh"])
@pytest.mark.parametrize("kind,n", [("dense", 1500), ("spanning", 3000), ("even", 65_535), ("even", 65_536)])
def test_pair_lists_past_the_kept_partners(sdlib, orc, op, kind, n):
    """Boxes with none to many more partners than are kept per box (16), a
    box over the whole domain with the lowest and the highest id, and either
    side of the tree's lane rule; a list that just fits, and one too short."""
    import torch
    rng = np.random.default_rng(n)
    c = rng.uniform(-1.0, 1.0, (n, 3)).astype(np.float32)
    h = np.full((n, 3), {"dense": 0.22, "spanning": 0.03, "even": 0.012}[kind], np.float32)
    if kind == "spanning":
        h[[0, n - 1]] = 3.0
    L = np.zeros((n, 4), np.float32)
    H = np.zeros((n, 4), np.float32)
    L[:, :3] = c - h
    H[:, :3] = c + h
    want = orc.aabb_pairs(L, H)
    lower = np.bincount((want >> np.uint64(32)).astype(np.int64), minlength=n)
    assert (lower.max() > 16) == (kind != "even") and 16 in lower or kind != "dense"
    pairs = sdlib.SweepAndPrune.pairs if op == "sap" else sdlib.BoundingVolumes.pairs
    lo, hi = torch.from_numpy(L).cuda(), torch.from_numpy(H).cuda()
    got, cnt, err = pairs(lo, hi, len(want))
    assert err == 0 and cnt == len(want)
    assert np.array_equal(got.cpu().numpy().view(np.uint64), want)
    assert pairs(lo, hi, len(want) - 1)[2] == sdlib._abi.SD_DEVERR_PAIR_OVERFLOW


@pytest.mark.parametrize("n", [2, 127, 128, 129, 512, 513, 640, 641, 1153, 5000])
@pytest.mark.parametrize("spread", [1.0, 1e-3, 0.0])
def test_tree_over_treelets(sdlib, orc, n, spread):
    """Trees around the sizes of a treelet (128 leaves) and of a block's
    window (512 + 128), with many equal codes, and nothing but equal codes."""
    import torch
    rng = np.random.default_rng(n)
    c = (rng.uniform(-1.0, 1.0, (n, 3)) * (np.where(rng.random((n, 1)) < 0.7, spread, 1.0) if spread else 0.0)).astype(np.float32)
    h = (rng.uniform(0.2, 1.0, (n, 3)) * (0.05 if spread == 1.0 else 2e-4)).astype(np.float32)
    if n > 1000:
        c += rng.integers(0, n // 50, (n, 1)).astype(np.float32) * (4.0 if spread else 0.0)
    if spread == 0.0:
        c[:, 0] = np.arange(n) * np.float32(3e-4)
        c[0, 0], c[n - 1, 0] = -1e4, 1e4  # the rest share one cell of the code
    L = np.zeros((n, 4), np.float32)
    H = np.zeros((n, 4), np.float32)
    L[:, :3] = c - h
    H[:, :3] = c + h
    want = orc.aabb_pairs(L, H)
    got, cnt, err = sdlib.BoundingVolumes.pairs(torch.from_numpy(L).cuda(), torch.from_numpy(H).cuda(), len(want) + 1)
    assert err == 0 and cnt == len(want)
    assert np.array_equal(got.cpu().numpy().view(np.uint64), want)


@pytest.mark.parametrize("n", [3, 4097, 32_767, 32_768, 32_769, 4_194_304, 4_194_305])
def test_pair_offsets_over_scan_sizes(sdlib, n):
    """Either side of the scan's one block (32,768) and of its two launches
    (2,048 tiles of 2,048): boxes in a row, each on the next one."""
    import torch
    x = torch.arange(n, dtype=torch.float32, device="cuda") * 2.0
    L = torch.zeros((n, 4), device="cuda")
    H = torch.ones((n, 4), device="cuda")
    L[:, 0], H[:, 0] = x, x + 2.0
    got, cnt, err = sdlib.SweepAndPrune.pairs(L, H, n)
    i = torch.arange(n - 1, device="cuda")
    assert err == 0 and cnt == n - 1 and torch.equal(got, (i << 32) | (i + 1))


@pytest.mark.parametrize("n,cols", [(255, 1), (256, 1), (257, 2), (700, 2), (3000, 1), (20_000, 8)])
def test_sweep_past_a_blocks_entries(sdlib, orc, n, cols):
    """Columns of entries around and over the 256 + 64 that a block holds, x
    windows of some and of all of them, more pairs than a block sets aside,
    and pairs whose boxes share two and four columns."""
    import torch
    rng = np.random.default_rng(n)
    c = rng.uniform(0.0, 1.0, (n, 3)).astype(np.float32)
    c[:, 1:] = 0.013 * rng.integers(0, cols, (n, 2)) + rng.uniform(0.0, 0.012, (n, 2))
    h = np.full((n, 3), 0.005, np.float32)
    h[:, 0] = 0.5 * np.where(rng.random(n) < 0.05, 0.6, 60.0 / n)
    L = np.zeros((n, 4), np.float32)
    H = np.zeros((n, 4), np.float32)
    L[:, :3] = c - h
    H[:, :3] = c + h
    want = orc.aabb_pairs(L, H)
    got, cnt, err = sdlib.SweepAndPrune.pairs(torch.from_numpy(L).cuda(), torch.from_numpy(H).cuda(), len(want) + 1)
    assert err == 0 and cnt == len(want)
    assert np.array_equal(got.cpu().numpy().view(np.uint64), want)


def _workspace(op, n, cap):
    """Bytes of the workspace that held both ways' partner lists, which a
    program may keep: it stays enough."""
    a = lambda x: (x + 255) // 256 * 256
    m = max(n, 1)
    sort = lambda k, passes: a(4 * (16 + 4 * 512 + passes * -(-k // 2048) * 512))
    scan = a(4 * (-(-(m + 1) // 2048) + 1))
    if op == "lbvh":
        return (4 * a(4 * m) + sort(m, 4) + a(32) + a(24 * 304) + a(8 * m) + a(8 * m) + a(4 * m) + 4 * a(16 * m) +
                a(4 * (m + 1)) + scan + 2 * a(64 * m) + a(16) + 2 * a(4 * (n + 1)) +
                2 * a(4 * (2 * cap + 1)))
    return (4 * a(4 * m) + sort(m, 4) + 4 * a(16 * m) + 3 * a(4 * (m + 1)) + scan + a(4 * (2 * cap + 1)) + a(16) +
            4 * a(16 * m) + sort(4 * m, 2) + a(64))


@pytest.mark.parametrize("op", ["sap", "lbvh", "process"])
@pytest.mark.parametrize("n", [1, 300, 5000, 100_003])
def test_workspaces_stay_enough(sdlib, orc, op, n):
    """A workspace of the size above is taken, and nothing is written past
    the size that the library asks for."""
    import ctypes as C
    import torch
    from stardust_gb300 import _abi
    rng = np.random.default_rng(n)
    L, H = np.zeros((n, 4), np.float32), np.zeros((n, 4), np.float32)
    c = rng.uniform(0.1, 0.9, (n, 3))
    L[:, :3], H[:, :3] = c - 0.5 * n ** (-1 / 3), c + 0.5 * n ** (-1 / 3)
    want = orc.aabb_pairs(L, H)
    cap = 0 if op == "process" else len(want)
    ask = C.c_uint64()
    _abi.call("sd_lbvh_scratch_bytes" if op == "lbvh" else "sd_sap_scratch_bytes", n, cap, C.byref(ask))
    kept = _workspace("lbvh" if op == "lbvh" else "sap", n, cap)
    buf = torch.full((max(kept, ask.value) + 4096,), 0xA5, dtype=torch.uint8, device="cuda")
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    lo, hi = torch.from_numpy(L).cuda(), torch.from_numpy(H).cuda()
    if op == "process":
        pos = torch.from_numpy(np.concatenate([c, np.full((n, 1), 0.01)], 1).astype(np.float32)).cuda()
        rows = torch.empty((n, 16), dtype=torch.int32, device="cuda")
        _abi.call("sd_sap_process_collisions", n, pos.data_ptr(), None, rows.data_ptr(), buf.data_ptr(), kept, st)
        assert torch.equal(rows, sdlib.SweepAndPrune.process_collisions(pos))
    else:
        out = torch.empty(max(cap, 1), dtype=torch.int64, device="cuda")
        cnt = torch.zeros(2, dtype=torch.int32, device="cuda")
        _abi.call(f"sd_{op}_pairs", n, lo.data_ptr(), hi.data_ptr(), out.data_ptr(), cap, cnt.data_ptr(), buf.data_ptr(),
                  kept, st)
        assert cnt.tolist() == [len(want), 0]
        assert np.array_equal(out.cpu().numpy().view(np.uint64)[:cap], want)
    assert (buf[ask.value:] == 0xA5).all()


@pytest.mark.parametrize("n", [287, 288, 289, 543, 544, 545])
def test_sweep_at_the_end_of_a_blocks_entries(sdlib, orc, n):
    """One column that ends at, before and behind the 256 + 32 entries that a
    block holds, and so for the second block; every box's window in x reaches
    past them."""
    import torch
    rng = np.random.default_rng(n)
    c = rng.uniform(0.0, 1.0, (n, 3)).astype(np.float32)
    h = np.array([1.0, 0.02, 0.02], np.float32)
    c[:, 1:] *= np.float32(0.03)
    L = np.zeros((n, 4), np.float32)
    H = np.zeros((n, 4), np.float32)
    L[:, :3] = c - h
    H[:, :3] = c + h
    want = orc.aabb_pairs(L, H)
    assert len(want) > 30 * n
    got, cnt, err = sdlib.SweepAndPrune.pairs(torch.from_numpy(L).cuda(), torch.from_numpy(H).cuda(), len(want))
    assert err == 0 and cnt == len(want)
    assert np.array_equal(got.cpu().numpy().view(np.uint64), want)


@pytest.mark.parametrize("op,n", [("sap", 50_001), ("lbvh", 5_001), ("lbvh", 70_001)])
def test_pairs_captured(sdlib, orc, op, n):
    """The operators in a caller's graph, where what a step clears is cleared
    by memsets and the launches are plain ones: replayed on new boxes and over
    a workspace that holds something else."""
    import ctypes as C
    import torch
    from stardust_gb300 import _abi
    rng = np.random.default_rng(n)
    boxes = []
    for _ in range(2):
        L, H = np.zeros((n, 4), np.float32), np.zeros((n, 4), np.float32)
        c = rng.uniform(0.0, 1.0, (n, 3))
        h = rng.uniform(0.2, 1.0, (n, 1)) * n ** (-1 / 3)
        L[:, :3], H[:, :3] = c - h, c + h
        boxes.append((L, H, orc.aabb_pairs(L, H)))
    cap = max(len(b[2]) for b in boxes)
    size = C.c_uint64()
    _abi.call(f"sd_{op}_scratch_bytes", n, cap, C.byref(size))
    scratch = torch.zeros(size.value, dtype=torch.uint8, device="cuda")
    lo, hi = (torch.zeros((n, 4), device="cuda") for _ in range(2))
    out = torch.zeros(cap, dtype=torch.int64, device="cuda")
    cnt = torch.zeros(2, dtype=torch.int32, device="cuda")
    graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=side):
        _abi.call(f"sd_{op}_pairs", n, lo.data_ptr(), hi.data_ptr(), out.data_ptr(), cap, cnt.data_ptr(),
                  scratch.data_ptr(), scratch.numel(), C.c_void_p(side.cuda_stream))
    for fill, (L, H, want) in zip((0xAB, 0x01, 0xFF), (*boxes, boxes[0])):
        lo.copy_(torch.from_numpy(L))
        hi.copy_(torch.from_numpy(H))
        scratch.fill_(fill)
        cnt.fill_(7)
        graph.replay()
        torch.cuda.synchronize()
        assert cnt.tolist() == [len(want), 0]
        assert np.array_equal(out.cpu().numpy().view(np.uint64)[:len(want)], want)
