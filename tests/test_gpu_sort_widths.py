"""The radix sort's passes at the edges of their digit widths and tiles (4096 keys), heavily skewed ids, and the
permutation kernel's record widths; bit-exact against numpy."""
import numpy as np
import pytest
import torch

from flexspmv_b200.python_wrapper.dynamic_replace_submodule import permute_edges, sort_edges_by_row

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [2, 3, 128, 129, 255, 256, 257, 65535, 65536, 65537, (1 << 24) + 1])
@pytest.mark.parametrize("n", [1, 31, 33, 4095, 4096, 4097, 3 * 4096 + 5])
def test_digit_widths_and_tiles(rows, n):
    rng = np.random.default_rng(rows + n)
    draws = {"uniform": rng.integers(0, rows, n), "last": np.full(n, rows - 1), "two": rng.choice([0, rows - 1], n),
             "descending": np.sort(rng.integers(0, rows, n))[::-1]}
    for what, ids in draws.items():
        for dtype in (np.int32, np.int64):
            perm, crow = sort_edges_by_row(torch.from_numpy(ids.astype(dtype)).cuda(), rows)
            assert np.array_equal(perm.cpu().numpy(), np.argsort(ids, kind="stable").astype(np.int32)), what
            want = np.searchsorted(np.sort(ids), np.arange(rows + 1)) if rows < 1 << 20 else None
            if want is not None:
                assert np.array_equal(crow.cpu().numpy(), want), what
            else:
                got = crow.cpu().numpy()
                assert got[0] == 0 and got[-1] == n and np.array_equal(np.diff(got).nonzero()[0], np.unique(ids)), what


@pytest.mark.parametrize("words", [1, 2, 3, 4, 6])
@pytest.mark.parametrize("n", [1, 1023, 1025, 70001])
@pytest.mark.parametrize("offset", [0, 1])
def test_permute_record_widths(words, n, offset):
    """``offset``: the source begins one word into an allocation, so wide records are not aligned to their width."""
    g = np.random.default_rng(n + words)
    base = torch.from_numpy(g.integers(-2 ** 31, 2 ** 31, n * words + 1).astype(np.int32)).cuda()
    src = base[offset:offset + n * words].view(n, words)
    perm = torch.from_numpy(g.permutation(n).astype(np.int32)).cuda()
    got = permute_edges(src, perm)
    assert torch.equal(got, src[perm.long()])


def test_counts_of_more_than_a_thousand_tiles_and_records_beyond_one_sweep():
    """4.3 M ids are 1050 tiles of counts (the scan over a digit's counts takes a second round from 1024 on), and 8-byte
    records beyond 2.4 M are the second sweep of the permutation's grid."""
    n, rows = 4_300_003, 70_001
    ids = np.random.default_rng(83).integers(0, rows, n)
    perm, ro = sort_edges_by_row(torch.from_numpy(ids).cuda(), rows)
    want = np.argsort(ids, kind="stable")
    assert np.array_equal(perm.cpu().numpy(), want)
    assert np.array_equal(ro.cpu().numpy(), np.searchsorted(ids[want], np.arange(rows + 1)))
    for dtype in (np.float64, np.float32):
        src = np.random.default_rng(89).random(n).astype(dtype)
        assert np.array_equal(permute_edges(torch.from_numpy(src).cuda(), perm).cpu().numpy(), src[want])


@pytest.mark.parametrize("rows,n", [(1 << 17, 2_999_999), (1 << 17, 3_000_000), ((1 << 17) + 1, 5 << 20), ((1 << 18) - 5, (5 << 20) + 1), (1 << 20, 3_000_001),
                                    (1 << 10, 200_003), ((1 << 9) - 1, 200_003)])
def test_lines_between_digit_widths(rows, n):
    """Two digits of nine bits between 3 M and 5 M ids of 17 and 18 bits, one of nine or ten, narrow ones elsewhere."""
    ids = np.random.default_rng(97).integers(0, rows, n)
    perm, ro = sort_edges_by_row(torch.from_numpy(ids.astype(np.int32)).cuda(), rows)
    want = np.argsort(ids, kind="stable")
    assert np.array_equal(perm.cpu().numpy(), want)
    assert np.array_equal(ro.cpu().numpy(), np.searchsorted(ids[want], np.arange(rows + 1)))
