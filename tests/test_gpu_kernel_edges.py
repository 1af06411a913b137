'''Sizes at which a kernel or the rule that picks it can go wrong: edges of
tiles and blocks, remainders, the smallest and the largest of a range.  Every
result is exact, against the oracle's restatement.'''

import numpy as np
import oracle
import pytest
from conftest import load_plan
from srdatalog_b200 import native
from srdatalog_b200 import workloads as W
from test_gpu_primitives import gpu_diff, gpu_merge, gpu_sort_unique, keys_with_bits

pytestmark = pytest.mark.gpu
torch = pytest.importorskip('torch')

TOP = np.uint64(0xFFFFFFFFFFFFFFFF)


# one block sorts up to 16,384 keys; above, blocks take at least 2,048 keys and
# tiles of at most 8,192; digits are 5 to 9 bits wide
@pytest.mark.parametrize('bits', [2, 13, 16, 19, 32])
@pytest.mark.parametrize('n', [2, 1023, 1025, 16_383, 16_384, 16_385, 40_961, 2_424_833])
def test_sort_unique_block_edges(n, bits):
  rng = np.random.default_rng(n + bits)
  k = keys_with_bits(rng, n, bits, dup_frac=0.2)
  assert np.array_equal(gpu_sort_unique(k, bits), oracle.sort_unique(k))


# a bitmap set sorts when the key space has at most 4,096 keys per input key and
# at most 2^28 in all, and the caller's scratch has room for it (33 MB at most);
# with the stated scratch it has that for small sets or many keys
@pytest.mark.parametrize('room', [0, 40 << 20])
@pytest.mark.parametrize('bits,n', [(1, 16_385), (5, 6001), (5, 20_000), (6, 20_000), (12, 6000), (12, 6001),
                                    (13, 16_384), (13, 16_385), (14, 65_535), (14, 65_536), (14, 3_000_000),
                                    (15, 3_000_000)])
@pytest.mark.parametrize('dense', [False, True])
def test_sort_unique_key_sets(bits, n, dense, room):
  rng = np.random.default_rng(n + bits)
  k = keys_with_bits(rng, n, bits)
  if dense:   # a block of the key space filled, the rest nearly empty
    k[: n - n // 16] = keys_with_bits(rng, n - n // 16, max(1, bits - 3))
  k[n // 2] = ((1 << bits) - 1) << 32 | ((1 << bits) - 1)
  assert np.array_equal(gpu_sort_unique(k, bits, room=room), oracle.sort_unique(k))


@pytest.mark.parametrize('n', [5000, 300_000])
def test_sort_unique_one_digit(n):
  '''Every key equal, then all but one (largest counters of a tile, keys of all ones).'''
  k = np.full(n, TOP, np.uint64)
  assert np.array_equal(gpu_sort_unique(k, 32), np.array([TOP]))
  k[n // 3] = 0
  assert np.array_equal(gpu_sort_unique(k, 32), np.array([0, TOP], np.uint64))
  for bits in (14, 16):   # the largest key of a bitmap set; all ones in 32-bit packed form
    top = np.full(n, (((1 << bits) - 1) << 32) | ((1 << bits) - 1), np.uint64)
    assert np.array_equal(gpu_sort_unique(top, bits), top[:1])
  assert np.array_equal(gpu_sort_unique(np.sort(keys_with_bits(np.random.default_rng(n), n, 7)), 7),
                        oracle.sort_unique(keys_with_bits(np.random.default_rng(n), n, 7)))


@pytest.mark.parametrize('bits,n', [(17, 100), (17, 5003), (32, 16_384), (5, 300_000), (13, 3_000_000), (16, 20_000)])
def test_sort_unique_refuses_little_scratch(bits, n):
  '''A region for the packed keys alone is too small, whichever path they take.'''
  k = torch.from_numpy(keys_with_bits(np.random.default_rng(n), n, bits).view(np.int64)).cuda()
  out, d_n = torch.full_like(k, -1), torch.full((1,), -1, dtype=torch.int64, device='cuda')
  size = 2 * n * (4 if bits <= 16 else 8)
  scratch = torch.empty(size, dtype=torch.uint8, device='cuda')
  rc = native.lib().srdl_sort_unique_u64(k.data_ptr(), n, bits, out.data_ptr(), d_n.data_ptr(), scratch.data_ptr(),
                                         size, torch.cuda.current_stream().cuda_stream)
  assert rc == 5 and int(d_n) == -1 and bool((out == -1).all())


@pytest.mark.parametrize('na,nb', [(1, 4), (2047, 2049), (2048, 2048), (31, 6000), (4096, 4096 * 16),
                                   (4096, 4096 * 16 + 1), (20_481, 700_000), (1_300_000, 2),
                                   # both sides of the line between streaming FULL and searching it
                                   (1_555_556, 1), (1_555_556, 3), (2_000_000, 2_000_000), (2_000_000, 2_000_001),
                                   (2_043_904, 4097), (2_043_905, 2047), (3_000_017, 6_500_076)])
def test_set_difference_tile_edges(na, nb):
  rng = np.random.default_rng(na + nb)
  u = np.unique(np.concatenate([keys_with_bits(rng, na + nb, 32), np.array([0, TOP], np.uint64)]))
  a = np.sort(rng.choice(u, min(na, len(u)), replace=False))
  b = np.sort(rng.choice(u, min(nb, len(u)), replace=False))
  a[0], a[-1] = u[0], u[-1]   # the smallest and the largest key there is
  for bb in (b, np.unique(np.append(b, u[0])), np.unique(np.append(b, u[-1])), b[b > a[len(a) // 2]]):
    assert np.array_equal(gpu_diff(a, bb), oracle.set_difference(a, bb))


@pytest.mark.parametrize('na,nb', [(1, 2047), (2048, 0), (2048, 2048), (2049, 4095), (1, 2_000_000),
                                   (2048 * 148 * 6, 5)])
@pytest.mark.parametrize('apart', [False, True])
def test_merge_tile_edges(na, nb, apart):
  rng = np.random.default_rng(na + 7 * nb)
  u = np.unique(keys_with_bits(rng, na + nb + 10, 28))[:na + nb]
  if not apart:
    rng.shuffle(u)
  a, b = np.sort(u[:na]), np.sort(u[na:])
  assert np.array_equal(gpu_merge(a, b), oracle.merge(a, b))


@pytest.mark.parametrize('n', [8191, 8192, 8193, 262_144, 262_145, 2_400_007])
def test_dump_piece_edges(n):
  '''Results read back in one small piece, in one large one and in several.'''
  rng = np.random.default_rng(n)
  k = np.unique(keys_with_bits(rng, n + n // 8 + 64, 20))
  k = rng.permutation(k)[:n]
  rows = np.stack([k >> np.uint64(32), k & np.uint64(0xFFFFFFFF)], 1).astype(np.uint32)
  with native.Database(load_plan('triangle')) as db:
    db.load_rows('KnowsInput', rows)
    db.run()
    for _ in range(2):
      assert np.array_equal(db.dump('Knows'), rows[np.argsort(k)])


@pytest.mark.parametrize('m', [4095, 4096, 4097, 16_384, 16_385, 120_000])
def test_count_scan_edges(m):
  '''Tables on both sides of the one-block count and scan.'''
  e = W.rmat_edges(13, 2 * m, seed=m)[:m]
  with native.Database(load_plan('triangle')) as db:
    db.load_rows('KnowsInput', e)
    db.run()
    assert db.count('TriangleJoin') == oracle.triangle_count(e)


@pytest.mark.parametrize('pivot_min', [1, 3, 64, 1 << 20])
@pytest.mark.parametrize('scale,draws', [(6, 3000), (12, 60_000)])
def test_pivot_rows_of_every_length(scale, draws, pivot_min):
  '''Count by shared-memory bitmaps: lists of any length, hubs that share their
  candidates among warps, and none at all.'''
  e = W.rmat_edges(scale, draws, seed=scale)
  with native.Database(load_plan('triangle')) as db:
    db.set_option('pivot_min', pivot_min)
    db.load_rows('KnowsInput', e)
    db.run()
    assert db.count('TriangleJoin') == oracle.triangle_count(e)


@pytest.mark.parametrize('n', [1500, 5000])
def test_pivot_hub_of_short_rows(n):
  '''A hub's rows on both sides of the shortest list that is staged (16), some
  without a whole quad and some empty, more of them than a block stages at once.'''
  i = np.arange(1, n, dtype=np.int64)
  own = np.concatenate([np.stack([i, i + d], 1)[(i % 41 >= d) & (i + d < n)] for d in range(1, 41)])
  hub = np.stack([np.zeros(n - 1, np.int64), i], 1)
  e = np.concatenate([hub, own]).astype(np.uint32)
  want = oracle.triangle_count(e)
  for pm in (1, 16, 1000):
    with native.Database(load_plan('triangle')) as db:
      db.set_option('pivot_min', pm)
      db.load_rows('KnowsInput', e)
      db.run()
      assert db.count('TriangleJoin') == want


def test_pivot_hub_of_many_pieces():
  '''One value whose rows make several million candidates.'''
  hub = np.stack([np.zeros(5000, np.uint32), np.arange(1, 5001, dtype=np.uint32)], 1)
  rng = np.random.default_rng(3)
  rest = rng.integers(1, 5001, (900_000, 2)).astype(np.uint32)
  rest = rest[rest[:, 0] < rest[:, 1]]
  e = np.unique(np.concatenate([hub, rest]), axis=0)
  counts = []
  for pm in (0, 16):
    with native.Database(load_plan('triangle')) as db:
      db.set_option('pivot_min', pm)
      db.load_rows('KnowsInput', e)
      db.run()
      counts.append(db.count('TriangleJoin'))
  assert counts[0] == counts[1] == oracle.triangle_count(e)


@pytest.mark.parametrize('pivot_min', [1, 20])
def test_pivot_rows_under_a_memory_limit(pivot_min):
  '''A limit that the run fits under without the pivot rows' scratch.'''
  e = W.rmat_edges(14, 350_000, seed=9)
  want = oracle.triangle_count(e)
  with native.Database(load_plan('triangle')) as db:
    db.set_option('bitmap_mb', 0)
    db.set_option('pivot_min', 0)
    db.load_rows('KnowsInput', e)
    db.set_option('mem_limit_mb', 1 << 12)
    db.run()
    limit = -(-db.mem_stats()['peak'] // (1 << 20))
    db.set_option('mem_limit_mb', limit)
    db.run()
    assert db.count('TriangleJoin') == want
    db.set_option('pivot_min', pivot_min)
    db.run()
    assert db.count('TriangleJoin') == want
    assert db.mem_stats()['peak'] <= limit << 20
    db.set_option('mem_limit_mb', 0)
    db.run()
    assert db.count('TriangleJoin') == want
