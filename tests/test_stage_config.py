"""Configuration codes survive the round trip through their fields."""
import pytest

from bbwadg_b200.solver import decode_config, encode_config

CTA = [w | o << 8 | p << 9 | e << 10 for w in (8, 16) for o in (0, 1) for p in (0, 1) for e in (0, 1)]
MATRIX = [8 | 1 << 8 | 1 << 10 | 1 << b for b in (11, 12)]


@pytest.mark.parametrize("code", CTA + MATRIX)
def test_round_trip(code):
    f = decode_config(code)
    assert f["code"] == code
    assert encode_config(f["warps"], f["ops_in_smem"], f["pipelined"], f["tile"]) == code
