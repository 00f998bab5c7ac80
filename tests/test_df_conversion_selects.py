"""to_df of csrc/df64.cuh as it stands, its range edges by selects instead of
a second path, restated in numpy (CPU): the same pairs as the two-path form of
test_df_conversion.py for every biased exponent and both signs."""
from __future__ import annotations

import numpy as np

from test_df_conversion import U32, _bits, _funnel29, to_df


def to_df_selects(v):
    lo32, hi32 = _bits(v)
    sign = hi32 & U32(0x80000000)
    de = (hi32 >> U32(20)) & U32(0x7FF)
    hb = (_funnel29(lo32, hi32) + U32(0x40000000)) | sign
    scale = (np.maximum(de, U32(948)) - U32(948)) << U32(23)
    hb = np.where(de < 897, sign, hb)
    nan = (de == 0x7FF) & (((hi32 & U32(0xFFFFF)) | lo32) != 0)
    hb = np.where(de > 1150, np.where(nan, sign | U32(0x7FC00000), sign | U32(0x7F800000)), hb)
    scale = np.where(de > 1150, U32(0), scale)
    r = (lo32 & U32(0x1FFFFFFF)).astype(np.int64)
    drop = np.maximum(np.floor(np.log2(np.maximum(r, 1))).astype(np.int64) - 23, 0)   # __int2float_rz
    rz = ((r >> drop) << drop).astype(np.float32)
    return hb.astype(U32).view(np.float32), np.where(sign != 0, -rz, rz) * scale.astype(U32).view(np.float32)


def test_same_pairs_over_all_exponents():
    rng = np.random.default_rng(8)
    mant = np.concatenate([rng.integers(0, 1 << 52, 60, dtype=np.uint64),
                           np.array([0, 1, (1 << 52) - 1, (1 << 29) - 1, 1 << 29, 1 << 28, 1 << 24], np.uint64)])
    e = np.arange(2048, dtype=np.uint64)
    b = (e[:, None] << np.uint64(52)) | mant[None, :]
    v = np.concatenate([b, b | np.uint64(1 << 63)]).reshape(-1).view(np.float64)
    with np.errstate(all="ignore"):
        hi, lo = to_df(v)
        hj, lj = to_df_selects(v)
    assert np.array_equal(hi.view(U32), hj.view(U32))
    assert np.array_equal(lo, lj)
