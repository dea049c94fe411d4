"""CPU check of the compaction's index arithmetic (gpu-preprocessor-ijoc_b200/csrc/
compact.cu), restated in numpy with small parts: the bits of the row starts and of the
kept ones over the entries, the byte by which a part learns of the row that it begins in
(set for the parts that begin inside a row, whatever it held before), the kept masks, the
kept entries before each part, and every kept row's new pointer from those two; two
matrices in one launch share the words, the second's behind the first's tiles."""
import numpy as np
import pytest

from test_tile_indexing import maps, plain_compact

BITS = 32


def last_bit(word):
    return int(word).bit_length() - 1


def compact_sides(sides, rounds, warps, rng):
    """`sides`: (ptr, idx, outer, inner) each; returns the new pointers and indices of each."""
    part = BITS * rounds
    tiles = [(len(idx) + part * warps - 1) // (part * warps) for _, idx, _, _ in sides]
    total_parts = sum(tiles) * warps
    starts = np.zeros(total_parts * rounds, dtype=np.uint64)   # zero at launch
    keeps = np.zeros(total_parts * rounds, dtype=np.uint64)
    part_kept = rng.random(total_parts) < 0.5                  # not cleared
    masks = rng.integers(0, 2**32, total_parts * rounds, dtype=np.uint64)
    out = []
    for side, (ptr, idx, outer, inner) in enumerate(sides):
        nnz, first = len(idx), (tiles[0] * warps if side else 0)
        words = first * rounds
        for r in range(len(ptr) - 1):   # compact_mark_rows
            a, e = int(ptr[r]), int(ptr[r + 1])
            if a == e:
                continue
            kept = outer[r] >= 0
            starts[words + a // BITS] |= np.uint64(1 << a % BITS)
            if kept:
                keeps[words + a // BITS] |= np.uint64(1 << a % BITS)
            for w in range(a // part + 1, (e + part - 1) // part):
                assert a < w * part < e
                part_kept[first + w] = kept
        before, count, new_idx = [], 0, []
        for w in range(tiles[side] * warps):   # compact_tiles, a warp
            length = max(0, min(part, nnz - w * part))
            carry = length > 0 and bool(part_kept[first + w])
            before.append(count)
            for k in range(rounds):
                at = words + w * rounds + k
                s, kp = (int(starts[at]), int(keeps[at])) if k * BITS < length else (0, 0)
                mask = 0
                for lane in range(BITS):
                    q = w * part + k * BITS + lane
                    up_to = s & ((2 << lane) - 1)
                    row_kept = bool(kp >> last_bit(up_to) & 1) if up_to else carry
                    if k * BITS + lane < length:
                        row = np.searchsorted(ptr, q, side="right") - 1
                        assert row_kept == (outer[row] >= 0)
                        if row_kept and inner[idx[q]] >= 0:
                            mask |= 1 << lane
                            new_idx.append(inner[idx[q]])
                if s:
                    carry = bool(kp >> last_bit(s) & 1)
                masks[at] = mask
                count += bin(mask).count("1")
        new_ptr = np.full(int((outer >= 0).sum()) + 1, -1, dtype=np.int64)
        new_ptr[-1] = count
        for r in range(len(ptr) - 1):   # compact_row_pointers
            a = int(ptr[r])
            if a < nnz:
                starts[words + a // BITS] = keeps[words + a // BITS] = 0
            if outer[r] < 0:
                continue
            if a >= nnz:
                new_ptr[outer[r]] = new_ptr[-1]
                continue
            w = a // part
            kept = before[w] + sum(bin(int(masks[words + q])).count("1") for q in range(w * rounds, a // BITS))
            new_ptr[outer[r]] = kept + bin(int(masks[words + a // BITS]) & ((1 << a % BITS) - 1)).count("1")
        out.append((new_ptr, np.array(new_idx, dtype=np.int64)))
    assert not starts.any() and not keeps.any(), "the bits are left set"
    return out


def matrix(lens, cols, rng):
    ptr = np.concatenate([[0], np.cumsum(lens)])
    return ptr, rng.integers(0, cols, size=int(ptr[-1]))


LAYOUTS = {
    "random": lambda rng: rng.integers(0, 12, size=60),
    "long": lambda rng: np.array([5, 700, 0, 1, 300]),
    "one row": lambda rng: np.array([257]),
    "empty runs": lambda rng: np.concatenate([np.zeros(9, int), rng.integers(0, 40, 12), np.zeros(30, int)]),
    "part edges": lambda rng: np.array([0, 64, 0, 64, 32, 32, 0, 0, 63, 1, 128, 0]),
    "none": lambda rng: np.zeros(4, int),
}


@pytest.mark.parametrize("second", LAYOUTS)
@pytest.mark.parametrize("first", LAYOUTS)
def test_parts_of_two_sides(first, second):
    rng = np.random.default_rng(len(first) * 100 + len(second))
    for rounds, warps in ((2, 1), (2, 2), (1, 4)):
        for kept in (0.2, 0.7, 1.0):
            sides = []
            for layout in (first, second):
                ptr, idx = matrix(LAYOUTS[layout](rng), 20, rng)
                sides.append((ptr, idx, maps(rng.random(len(ptr) - 1) < kept), maps(rng.random(20) < kept)))
            for (ptr, idx, outer, inner), got in zip(sides, compact_sides(sides, rounds, warps, rng)):
                want = plain_compact(ptr, idx, outer, inner)
                assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
