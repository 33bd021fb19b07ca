"""Difflists decoded in shared memory: groups of one-byte, two-byte and longer
id gaps, group and record ends at every remainder, zero and padded deltas, ids past
the samples, several warps per record, and rows too long for shared memory."""
import numpy as np
import pytest

from gnomon_b200 import synth
from gnomon_b200.pgen import decode_to_device
from oracle import pgen_oracle
from test_gpu_pgen import device_rows
from test_pgen import expected_rows

pytestmark = pytest.mark.gpu


def file_of(n, lists):
    """A 2-bit record, then per id list an LD record (types 2 and 3 in turn) against
    it and a fill record (types 4, 6, 7 in turn) with the same difflist."""
    rng = np.random.default_rng(n)
    first = rng.integers(0, 4, n).astype(np.uint8)
    swap = np.array([2, 1, 0, 3], np.uint8)
    cats, types, recs = [first], [0], [None]
    pad = np.zeros((n + 3) // 4 * 4, np.uint8)
    pad[:n] = first
    q = pad.reshape(-1, 4)
    recs[0] = (q[:, 0] | q[:, 1] << 2 | q[:, 2] << 4 | q[:, 3] << 6).astype(np.uint8).tobytes()
    for j, ids in enumerate(lists):
        vals = rng.integers(0, 4, len(ids)).astype(np.uint8)
        body = synth._difflist_bytes(np.asarray(ids, np.int64), vals, n)
        ld = first.copy()
        ld[ids] = vals                    # type 3 swaps the patched row
        cats.append(swap[ld] if j % 2 else ld)
        types.append(3 if j % 2 else 2)
        recs.append(body)
    for j, ids in enumerate(lists):       # after the LD records, which diff against record 0
        vals = rng.integers(0, 4, len(ids)).astype(np.uint8)
        kind = (4, 6, 7)[j % 3]
        row = np.full(n, {4: 0, 6: 2, 7: 3}[kind], np.uint8)
        row[ids] = vals
        cats.append(row)
        types.append(kind)
        recs.append(synth._difflist_bytes(np.asarray(ids, np.int64), vals, n))
    return synth._pgen_file(n, types, recs), np.array(cats)


@pytest.mark.parametrize("n", [1, 17, 63, 64, 65, 255, 2_000, 50_001, 300_000, 819_200, 819_201])
def test_gaps_and_ends(cuda, n):
    rng = np.random.default_rng(7 * n)
    lists = [[], [n - 1], list(range(n))[:200]]
    for count in (1, 2, 63, 64, 65, 127, 128, 129, 191, 192, 193, 2_048, 2_049, 4_160):
        if count <= n:
            lists.append(np.sort(rng.choice(n, count, replace=False)))
    for gap in (1, 126, 127, 128, 129, 16_383, 16_384, 16_385):   # edges of one and two bytes
        ids = np.arange(0, n, gap)[:500]
        lists.append(ids)
        mixed = np.cumsum(rng.choice([1, 2, gap], 700))            # one- and multi-byte groups
        lists.append(mixed[mixed < n])
    data, cats = file_of(n, lists)
    got = device_rows(data, n)
    np.testing.assert_array_equal(got, expected_rows(cats))
    if n <= 50_001:
        np.testing.assert_array_equal(got, pgen_oracle.decode_to_bed(data))


@pytest.mark.parametrize("at", [1, 8, 30, 62, 63])
@pytest.mark.parametrize("what", ["zero", "next group", "unfinished"])
def test_malformed_deltas(cuda, at, what):
    """A group of one-byte deltas with a zero, one that runs into the next group, and
    one whose last byte goes on: an error, from whichever lane holds it."""
    n = 5_000
    ids = np.arange(3, 3 + 7 * 192, 7)
    data, _ = file_of(n, [ids])
    buf = bytearray(data)
    body = synth._difflist_bytes(ids, np.random.default_rng(n).integers(0, 4, len(ids)), n)
    deltas = len(body) - 189                      # three groups of 63 one-byte deltas, last
    rec = len(buf) - 2 * len(body) + deltas       # the LD record's deltas
    assert bytes(buf[rec:rec + 189]) == b"\x07" * 189
    buf[rec + at - 1] = {"zero": 0, "next group": 120, "unfinished": 0x87}[what]
    if what == "next group":
        buf[rec + at % 63] = 120
        buf[rec + (at + 5) % 63] = 120
        buf[rec + (at + 9) % 63] = 120
    with pytest.raises(Exception, match="malformed"):
        decode_to_device(bytes(buf))
