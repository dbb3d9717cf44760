"""The element offsets of a chunk record's tensor-core parts: every two bytes before the decay belong to one element."""
from kda_ascendc_b200 import layout as L


def test_record_parts_tile_the_record():
    wq, kg, aq = L._wq_index("cpu"), L._kg_index("cpu"), L._aq_index("cpu")
    at = [o + i for o, idx in ((L.REC_W, wq), (L.REC_QG, wq), (L.REC_KGH, kg), (L.REC_KGL, kg), (L.REC_AQK, aq), (L.REC_AQL, aq))
          for i in idx.reshape(-1).tolist()]
    assert sorted(at) == list(range(0, L.REC_DEC, 2))


def test_eight_rows_of_a_matrix_lie_in_different_banks():
    """What one ldmatrix pass reads (eight rows, 16 bytes each) covers all 32 banks."""
    wq, kg, aq = L._wq_index("cpu"), L._kg_index("cpu"), L._aq_index("cpu")
    for rows in (wq[:8, 0], wq[8:, 72], kg[0, 24:32], aq[8:, 8]):
        assert len({int(x) % 128 // 16 for x in rows}) == 8


def test_later_parts_tile_the_record():
    xb, v, dec2 = L._xb_index("cpu"), 2 * L._swizzle_index("cpu"), 4 * L._dec2_index("cpu")
    at = [o + i for o, idx in ((L.REC_XBH, xb), (L.REC_XBL, xb), (L.REC_V, v)) for i in idx.reshape(-1).tolist()]
    at += [L.REC_DEC2 + i + half for i in dec2.tolist() for half in (0, 2)]
    assert sorted(at) == list(range(L.REC_XBH, L.REC_USED_BYTES, 2))
    assert len({int(x) % 128 // 16 for x in xb[:8, 0]}) == 8 and len({int(x) % 128 // 16 for x in xb[8:, 8]}) == 8
