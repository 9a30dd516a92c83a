"""The serving top-k's filter pass (kernel variant 6) at the edges of its tiles,
thresholds and row blocks: corpora around one 256-code tile and around the
sample of the first threshold, one large enough for the second threshold, row
counts around the MMA's column steps and the 256-row blocks, nibble and byte
codes, reductions of one block and of many, zero rows and rows of very
different norms.  Results equal the stable argsort of the oracle's
distances bit for bit, and no candidate lies outside the pass's error bound."""
import numpy as np
import pytest

import oracle as O
import turboquant as tq

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,bits,n", [(64, 4, 1), (32, 4, 255), (100, 8, 256), (384, 4, 257), (1000, 3, 3000),
                                        (128, 8, 8191), (128, 2, 8193), (768, 8, 12_000), (64, 4, 340_000)])
@pytest.mark.parametrize("m,k", [(1, 1), (31, 10), (33, 16), (129, 10), (300, 10)])
def test_filter_edges(cuda_ok, dim, bits, n, m, k):
    rng = np.random.default_rng(dim + 3 * bits + n + m)
    X = (rng.standard_normal((n, dim)) * rng.uniform(0.5, 2.0, (n, 1))).astype(np.float32)
    X[n // 3] = 0.0
    Q = (rng.standard_normal((m, dim)) * rng.uniform(1e-2, 1e2, (m, 1))).astype(np.float32)
    Q[m // 2] = 0.0 if m > 1 else Q[m // 2]
    space, o = tq.TurboQuantSpace(dim, bits), O.OracleSpace(dim, bits)
    codes = space.encode_batch(X)
    ref = o.distance_m_to_n(Q, codes)
    idx = np.argsort(ref, axis=1, kind="stable")[:, :k]
    ix = space.index(codes)
    try:
        with ix.serve(k=k, max_rows=384, slots=1, kernel_variant=6) as sv:
            D, I = sv.submit(Q).wait()
            st = sv.stats()
    finally:
        ix.close()
    w = idx.shape[1]
    np.testing.assert_array_equal(I[:, :w], idx)
    np.testing.assert_array_equal(D[:, :w].view(np.uint32),
                                  np.take_along_axis(ref, idx, 1).astype(np.float32).view(np.uint32))
    assert np.all(I[:, w:] == -1)
    assert st["bound_violations"] == 0


@pytest.mark.parametrize("order", ["by cluster", "round robin"])
def test_storage_order_leaves_no_more_rows_open(cuda_ok, order):
    """Fifty clusters of 6,000 codes, a query near each: the filter's thresholds come
    from a sample that must not depend on the order the corpus is stored in.  Stored
    by cluster or round robin, at most a tenth more of the rows take the exact
    fallback than with the same corpus shuffled, and the results are the same."""
    rng = np.random.default_rng(11)
    dim, bits, per, groups, k = 64, 8, 6000, 50, 10
    n = per * groups
    centres = rng.standard_normal((groups, dim)).astype(np.float32)
    label = np.repeat(np.arange(groups), per) if order == "by cluster" else np.tile(np.arange(groups), per)
    X = (centres[label] + 0.3 * rng.standard_normal((n, dim))).astype(np.float32)
    Q = (centres + 0.3 * rng.standard_normal((groups, dim))).astype(np.float32)
    space, o = tq.TurboQuantSpace(dim, bits), O.OracleSpace(dim, bits)
    codes = space.encode_batch(X)
    ref = o.distance_m_to_n(Q, codes)
    idx = np.argsort(ref, axis=1, kind="stable")[:, :k]

    def search(c):
        ix = space.index(c)
        try:
            with ix.serve(k=k, max_rows=128, slots=1, kernel_variant=6) as sv:
                D, I = sv.submit(Q).wait()
                return D, I, sv.stats()["fallback_rows"]
        finally:
            ix.close()

    D, I, stored = search(codes)
    np.testing.assert_array_equal(I, idx)
    np.testing.assert_array_equal(D, np.take_along_axis(ref, idx, 1).astype(np.float32))
    perm = rng.permutation(n)
    D2, _, shuffled = search(codes[perm])
    np.testing.assert_array_equal(np.sort(D2, axis=1), np.sort(D, axis=1))
    print(f"{order}: {stored} open rows, {shuffled} shuffled")
    assert stored <= shuffled + groups // 10


def test_only_servers_that_may_filter_hold_its_buffers(cuda_ok):
    """The filter's buffers are 64 KB a query row: servers of another kernel variant
    do not hold them, and a server that tunes gives up the filter rather than slots
    where memory is short."""
    import torch

    rng = np.random.default_rng(2)
    space = tq.TurboQuantSpace(64, 4)
    codes = space.encode_batch(rng.standard_normal((3000, 64)).astype(np.float32))
    ix = space.index(codes)
    rows, slots = 4096, 8
    used = {}
    try:
        for variant in (4, 6):
            torch.cuda.synchronize()
            before = torch.cuda.mem_get_info()[0]
            with ix.serve(k=16, max_rows=rows, slots=2, kernel_variant=variant):
                used[variant] = before - torch.cuda.mem_get_info()[0]
        assert used[6] - used[4] >= 2 * rows * 64 * 1024, used
        # room for the slots themselves, by the server's own estimate, but not for the
        # filter's 270 MB each as well
        per_slot = rows * (64 * 4 + 130 * 4 + 128 * 4 + 16 * 12 + 32 * 12 + 300 * 16 * 8) + (32 << 20)
        leave = 2 * slots * per_slot + (512 << 20)
        fill = torch.empty(max(0, torch.cuda.mem_get_info()[0] - leave), dtype=torch.uint8, device="cuda")
        with ix.serve(k=16, max_rows=rows, slots=slots) as sv:
            assert sv.stats()["slots"] == slots
            assert all(b["variant"] != 6 for b in sv.tuning())
        del fill
    finally:
        ix.close()
        torch.cuda.empty_cache()
