"""Which prompts have blocks of two query tiles (the rule of attention_tc.cu, which runs on the host; no GPU)."""
import ctypes

import pytest

from photon_infer_b200.csrc.build import load_module


@pytest.mark.parametrize("keys,window,tiles_per_seq,tiles,pairs,two", [
    # long contexts, however few the tiles
    (14400, 0, 2, 16, 8, True), (4160, 0, 2, 16, 8, True), (16384, 0, 64, 512, 256, True), (4400, 0, 13, 416, 224, True),
    # few tiles behind 2,048 keys (40 and 42 us, 48 and 49)
    (2112, 0, 2, 16, 8, False), (2560, 0, 13, 104, 56, False),
    # one tile a request
    (1664, 0, 1, 16, 16, True), (640, 0, 1, 16, 16, False), (14353, 2048, 1, 8, 8, True), (14353, 1024, 1, 8, 8, False),
    # more tiles than multiprocessors (50 and 49, 33 and 34, 40 and 42), than two on each (54 and 50, 67 and 69)
    (2560, 0, 32, 256, 128, True), (1536, 0, 32, 256, 128, False), (2048, 0, 16, 256, 128, False), (2048, 0, 64, 512, 256, True),
    (2048, 0, 342, 684, 342, False),
    # short portions beside requests with long tables (12 and 17, 27 and 30)
    (300, 0, 5, 40, 24, False), (1093, 0, 27, 216, 112, False),
    # windows (22 and 30, 34 and 41, 46 and 48, 160 and 153, 76 and 79); one that nothing falls out of
    (2048, 128, 64, 512, 256, False), (16384, 512, 64, 512, 256, False), (10240, 1024, 64, 512, 256, False),
    (10240, 4096, 64, 512, 256, True), (8704, 4096, 13, 104, 56, False), (2048, 4096, 64, 512, 256, True)])
def test_two_tiles_where_they_are_faster(keys, window, tiles_per_seq, tiles, pairs, two):
    rule = load_module("attention_tc", {"HEAD_DIM": 128}).photon_attention_tc_two_tiles
    rule.argtypes, rule.restype = [ctypes.c_long, ctypes.c_int, ctypes.c_int, ctypes.c_long, ctypes.c_long, ctypes.c_int], ctypes.c_int
    assert bool(rule(keys, window, tiles_per_seq, tiles, pairs, 148)) == two
