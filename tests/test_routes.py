"""CPU tests of the rules that pick an attention call's schedule, a GEMM's tile shape and what a thread block of the pre-pass takes
(kiln_b200/csrc/routes.h, plain C++)."""
import ctypes

import pytest

import util_routes

WHOLE, BALANCED, KEYS = 0, 1, 2
SMS = 148

# Device time (us) of one call on a B200, fp16 operands in place, inside a CUDA graph: whole items, balanced schedule, keys split
# over both streams (None: the schedule does not exist there)
MEASURED = [  # B, Tq, Tk, H, whole, balanced, keys
    (1, 128, 4096, 16, 48.4, 33.9, 35.4), (1, 256, 4096, 16, 61.3, 37.6, 36.0), (1, 128, 8192, 16, 91.3, 39.9, 66.0), (1, 256, 16384, 4, 226.6, 87.8, 125.7),
    (1, 128, 16384, 16, 176.6, 52.2, 126.9), (1, 4096, 4096, 2, 61.5, 35.3, 36.9), (1, 4096, 4096, 4, 63.3, 46.4, 39.0), (1, 2000, 2000, 3, 34.0, 30.2, 20.9),
    (2, 2000, 2000, 2, 34.2, 29.3, 21.4), (1, 2048, 2048, 8, 35.1, 31.1, 23.0), (1, 1024, 1024, 16, 20.5, 25.1, 14.6), (1, 1152, 1152, 16, 22.9, 26.2, 15.6),
    (1, 1024, 4096, 16, 63.0, 46.6, 39.1), (1, 1024, 8192, 16, 119.3, 73.0, 70.7), (1, 512, 2048, 16, 34.1, 29.1, 21.4), (1, 512, 4096, 16, 61.6, 35.3, 36.9),
    (1, 512, 8192, 16, 117.9, 51.3, 67.5), (1, 2048, 4096, 2, 61.3, 37.3, 35.9), (1, 4096, 512, 4, 13.4, None, 10.2), (1, 256, 2048, 16, 33.6, None, 20.7),
    (1, 128, 3000, 32, 38.1, 27.5, 28.2), (1, 2304, 4096, 8, 62.6, 47.8, 39.1), (1, 1500, 1500, 12, 28.0, 28.5, 18.9), (1, 1, 8192, 32, 91.2, 45.6, 66.5),
    (1, 128, 4096, 148, 57.3, 58.3, 52.9), (1, 1280, 1280, 16, 25.8, 29.0, 28.7), (1, 2048, 2048, 16, 36.9, 43.8, 42.7), (1, 2560, 2560, 16, 81.3, 58.1, 71.8),
    (1, 1280, 4096, 16, 66.5, 50.5, 71.4), (1, 1408, 8192, 16, 124.0, 94.1, 133.2)]

# Device time (us) of a projection on a B200, inside a CUDA graph, with three widths forced in turn: 256, 224 and 192 columns, or where N is no
# multiple of 256 128 (single CTAs), 224 and 192; medians of single calls with pauses between them, and of calls without a pause (under the
# power cap; those differ by up to 8 % from run to run)
WIDTHS = [  # epilogue, M, N, K, single calls, sustained
    ('GELU16', 512, 8192, 2048, (21.2, 19.1, 25.9), (22.2, 20.0, 27.5)), ('GELU16', 768, 8192, 2048, (32.4, 28.0, 26.6), (35.6, 30.0, 28.5)),
    ('GELU16', 1024, 8192, 2048, (33.8, 29.4, 35.2), (38.4, 32.9, 40.0)), ('GELU16', 1280, 8192, 2048, (45.1, 37.9, 36.9), (53.1, 42.9, 40.9)),
    ('GELU16', 1536, 8192, 2048, (46.4, 40.6, 45.1), (54.8, 44.9, 51.5)), ('GELU16', 2048, 8192, 2048, (58.7, 52.2, 56.6), (71.7, 58.5, 64.0)),
    ('GELU16', 2304, 8192, 2048, (61.8, 61.4, 64.5), (72.6, 69.3, 74.9)), ('GELU16', 2816, 8192, 2048, (76.1, 73.7, 76.8), (88.8, 82.0, 87.7)),
    ('GELU16', 3072, 8192, 2048, (85.3, 77.5, 80.9), (106.0, 84.6, 89.2)), ('GELU16', 3456, 8192, 2048, (98.0, 89.1, 96.3), (115.4, 90.9, 107.9)),
    ('GELU16', 3600, 8192, 2048, (102.1, 96.9, 100.0), (121.2, 106.4, 109.5)), ('GELU16', 3840, 8192, 2048, (103.1, 98.0, 101.4), (122.4, 107.0, 110.2)),
    ('GELU16', 4096, 8192, 2048, (107.2, 102.4, 109.6), (123.2, 108.4, 122.3)), ('GELU16', 4352, 8192, 2048, (117.1, 111.3, 113.7), (140.9, 121.8, 124.8)),
    ('GELU16', 4608, 8192, 2048, (121.2, 115.0, 122.5), (144.2, 124.3, 137.8)), ('GELU16', 5120, 8192, 2048, (134.8, 127.0, 134.8), (162.9, 139.5, 151.0)),
    ('GELU16', 5632, 8192, 2048, (149.2, 140.3, 146.8), (177.0, 148.5, 161.1)), ('GELU16', 6912, 8192, 2048, (181.1, 174.8, 180.6), (205.6, 185.2, 193.7)),
    ('GELU16', 8192, 8192, 2048, (213.3, 202.9, 214.4), (242.7, 211.8, 231.6)), ('RESID', 1280, 2048, 2048, (19.1, 17.8, 16.0), (17.9, 16.5, 15.0)),
    ('RESID', 1280, 2048, 8192, (50.9, 46.4, 41.3), (55.1, 49.4, 43.6)), ('RESID', 1536, 2048, 2048, (19.8, 18.1, 16.4), (18.5, 17.1, 15.7)),
    ('RESID', 1536, 2048, 8192, (52.6, 46.8, 42.3), (60.3, 52.5, 46.3)), ('RESID', 1792, 2048, 2048, (19.8, 18.4, 23.2), (19.7, 18.2, 23.8)),
    ('RESID', 1792, 2048, 8192, (51.9, 48.5, 69.0), (59.5, 52.6, 82.8)), ('RESID', 2048, 2048, 2048, (20.1, 24.6, 24.9), (20.2, 25.1, 25.2)),
    ('RESID', 2048, 2048, 8192, (53.2, 76.5, 70.0), (57.9, 90.2, 81.5)), ('RESID', 2304, 2048, 2048, (20.8, 28.0, 25.6), (21.9, 29.8, 27.0)),
    ('RESID', 2304, 2048, 8192, (56.3, 80.2, 73.0), (64.0, 101.9, 89.2)), ('RESID', 2560, 2048, 2048, (30.7, 28.3, 26.3), (31.8, 29.1, 26.6)),
    ('RESID', 2560, 2048, 8192, (88.7, 81.6, 75.8), (107.4, 94.7, 83.7)), ('RESID', 2816, 2048, 2048, (31.1, 28.7, 26.6), (33.1, 30.2, 27.8)),
    ('RESID', 2816, 2048, 8192, (90.1, 84.0, 79.5), (109.9, 97.1, 85.8)), ('RESID', 3456, 2048, 2048, (31.7, 29.7, 34.1), (36.2, 33.5, 39.1)),
    ('RESID', 3456, 2048, 8192, (96.9, 94.9, 107.2), (118.1, 104.4, 133.1)), ('RESID', 3840, 2048, 2048, (32.8, 34.1, 35.8), (35.5, 37.9, 39.1)),
    ('RESID', 3840, 2048, 8192, (102.0, 116.4, 112.6), (115.4, 143.9, 129.1)), ('RESID', 4096, 2048, 2048, (33.1, 37.2, 36.2), (37.2, 43.1, 41.0)),
    ('RESID', 4096, 2048, 8192, (105.5, 121.5, 116.4), (120.1, 149.9, 133.4)), ('RESID', 4352, 2048, 2048, (33.8, 39.2, 36.9), (38.1, 45.8, 41.7)),
    ('RESID', 4352, 2048, 8192, (109.2, 128.3, 121.9), (124.7, 160.3, 135.2)), ('RESID', 4608, 2048, 2048, (34.1, 39.6, 37.5), (39.1, 46.8, 42.7)),
    ('RESID', 4608, 2048, 8192, (113.0, 132.8, 125.6), (126.9, 163.5, 143.4)), ('RESID', 5120, 2048, 2048, (43.4, 40.6, 39.2), (51.5, 46.8, 43.5)),
    ('RESID', 5120, 2048, 8192, (142.0, 140.6, 134.5), (179.8, 158.9, 139.3)), ('RESID', 6144, 2048, 2048, (45.7, 49.2, 48.5), (53.4, 59.0, 55.5)),
    ('RESID', 6144, 2048, 8192, (158.0, 173.4, 167.2), (180.8, 203.6, 182.6)), ('RESID', 6912, 2048, 2048, (48.8, 53.2, 54.6), (56.5, 63.6, 66.8)),
    ('RESID', 6912, 2048, 8192, (170.3, 191.0, 196.8), (191.2, 221.2, 236.2)), ('RESID', 8192, 2048, 2048, (59.4, 63.1, 61.1), (69.2, 74.2, 69.1)),
    ('RESID', 8192, 2048, 8192, (213.7, 228.4, 219.1), (244.7, 263.3, 233.1)), ('F16', 1536, 8192, 2048, (40.3, 38.6, 42.0), (47.0, 43.8, 48.8)),
    ('F16', 3456, 8192, 2048, (87.7, 85.7, 90.5), (105.2, 95.7, 104.8)), ('F16', 3840, 8192, 2048, (92.5, 94.9, 95.2), (106.7, 108.0, 106.2)),
    ('F16', 4352, 8192, 2048, (105.5, 107.5, 107.5), (123.3, 123.0, 120.5)), ('F32', 1536, 8192, 2048, (43.4, 41.6, 45.7), (52.0, 48.4, 54.6)),
    ('F32', 3456, 8192, 2048, (95.6, 93.2, 99.3), (111.9, 103.5, 115.1)), ('F16', 1537, 2056, 64, (5.1, 6.8, 7.8), (4.8, 6.5, 7.5)),
    ('F32', 1300, 2048, 64, (7.5, 7.2, 7.2), (7.2, 6.8, 6.5)), ('F32', 1300, 2048, 128, (7.8, 7.5, 7.2), (7.5, 7.2, 6.8)),
    ('F32', 1300, 2048, 256, (8.5, 8.2, 7.8), (7.9, 7.6, 7.5)), ('F32', 1300, 2048, 512, (9.9, 9.2, 8.9), (9.2, 8.8, 8.3)),
    ('F32', 1300, 2048, 1024, (12.6, 11.9, 10.9), (11.9, 10.9, 10.2)), ('F16', 1537, 2056, 128, (5.5, 7.2, 8.2), (5.0, 6.6, 7.7)),
    ('F16', 1537, 2056, 256, (6.1, 7.8, 8.5), (5.6, 7.2, 8.2)), ('F16', 1537, 2056, 512, (8.5, 8.9, 9.9), (7.7, 8.3, 9.6)),
    ('F16', 1537, 2056, 1024, (11.3, 11.3, 13.6), (10.2, 10.6, 12.6)), ('F16', 1537, 2056, 2048, (17.8, 16.7, 21.2), (17.1, 15.9, 21.0)),
    ('F16', 1536, 1928, 2048, (17.4, 16.4, 15.4), (17.1, 16.0, 14.6)), ('F16', 1536, 1928, 512, (8.2, 8.9, 8.5), (7.6, 8.2, 7.9)),
    ('RESID', 1536, 2048, 64, (8.5, 8.2, 7.8), (8.2, 7.6, 7.5)), ('RESID', 1536, 2048, 128, (8.9, 8.5, 8.2), (8.5, 7.9, 7.5)),
    ('RESID', 1536, 2048, 256, (9.6, 9.2, 8.5), (9.2, 8.5, 8.2)), ('RESID', 1536, 2048, 512, (10.9, 10.2, 9.6), (10.4, 9.6, 9.2)),
    ('RESID', 1536, 2048, 1024, (13.7, 12.6, 11.9), (12.9, 11.9, 10.9)), ('GELU16', 1536, 8192, 64, (19.1, 17.1, 19.8), (18.2, 16.2, 19.1)),
    ('GELU16', 1536, 8192, 256, (20.8, 18.8, 21.5), (19.9, 17.8, 20.6)), ('GELU16', 1536, 8192, 512, (23.6, 21.5, 24.6), (23.0, 20.6, 23.9)),
    ('GELU16', 1536, 8192, 1024, (31.4, 26.3, 29.4), (34.0, 27.9, 31.1)), ('GELU16', 512, 8192, 64, (9.6, 8.5, 11.6), (8.9, 7.9, 10.9)),
    ('GELU16', 512, 8192, 256, (10.6, 9.6, 12.3), (9.9, 8.9, 11.9)), ('GELU16', 512, 8192, 512, (12.3, 10.9, 13.7), (11.3, 10.2, 12.9)),
    ('GELU16', 512, 8192, 1024, (15.4, 14.0, 17.1), (14.2, 12.7, 16.1)), ('F16', 4096, 1000, 2048, (19.1, 24.2, 22.9), (18.9, 24.4, 22.8)),
    ('F32', 4096, 3000, 2048, (52.2, 45.7, 44.7), (61.0, 53.4, 50.6)), ('F16', 8192, 6144, 2048, (144.7, 149.2, 147.8), (165.5, 170.1, 163.1)),
    ('F16', 1000, 3080, 1024, (11.3, 11.6, 10.9), (10.4, 10.6, 9.9)),
    ('F32', 1100, 8192, 1024, (25.9, 24.2, 23.2), (28.3, 26.2, 24.7)), ('F16', 1100, 8192, 1024, (22.9, 21.8, 20.8), (25.5, 23.3, 22.5)),
    ('F16', 2000, 4096, 1024, (18.1, 19.5, 19.5), (18.5, 20.2, 20.2)), ('RESID', 1100, 8192, 1024, (29.4, 28.0, 27.0), (31.5, 29.7, 28.2)),
    ('GELU16', 1100, 8192, 1024, (30.0, 24.9, 23.9), (32.2, 26.0, 24.7)), ('F32', 1100, 8168, 1024, (24.6, 24.2, 23.2), (26.6, 26.4, 25.2)),
    ('F16', 1100, 8168, 1024, (22.4, 22.2, 21.2), (23.9, 24.0, 23.1)), ('GELU16', 1100, 8168, 1024, (27.0, 25.3, 24.2), (28.6, 26.4, 25.4))]

@pytest.fixture(scope="module")
def rules():
    return util_routes.rules()


@pytest.fixture(scope="module")
def route(rules):
    return rules.route


@pytest.mark.parametrize("case", MEASURED, ids=[f"{b}x{q}x{k}x{h}" for b, q, k, h, *_ in MEASURED])
def test_the_schedule_taken_is_the_fastest_measured_one(route, case):
    """Within 3 %, what one side differs by from run to run."""
    B, Tq, Tk, H, *us = case
    taken = route(B, Tq, Tk, H, SMS, 1, 1)
    assert us[taken] is not None and us[taken] <= 1.03 * min(t for t in us if t is not None)


def test_restrictions(route):
    assert route(1, 128, 16384, 16, SMS, 1, 0) == KEYS and route(1, 2560, 2560, 16, SMS, 1, 0) == WHOLE      # no room for partial results
    assert route(1, 1024, 1024, 16, SMS, 0, 1) == WHOLE and route(1, 4096, 4096, 2, SMS, 0, 1) == BALANCED   # a call with peers
    for Tq in (1, 128, 129, 4096):
        assert route(1, Tq, 128, 1, SMS, 1, 1) == WHOLE                                                      # one key block: one stream has none


def test_projections_sum_in_one_order_whether_they_share_a_launch_or_not(rules):
    """The number of k ranges is the same for one, two and three segments; a split that is chosen has room for all its clusters."""
    splits = set()
    for mc2, mc4 in ((74, 37), (70, 32), (0, 0)):
        for M in (1, 77, 128, 129, 200, 256, 300, 512, 700, 1000, 1536, 4096):
            for N in (128, 256, 384, 1920, 2048):
                for ksteps in (2, 16, 32, 33, 128):
                    shapes = [rules.gemm(M, N, ksteps, n, 1, mc2, mc4) for n in (1, 2, 3)]
                    assert len({g & 7 for g in shapes}) == 1, (M, N, ksteps, shapes)
                    splits.add(shapes[0] & 7)
                    for n, g in zip((1, 2, 3), shapes):
                        tile, split = (256 if g & 8 else 128), g & 7
                        assert split == 1 or -(-M // tile) * -(-N // tile) * n <= (mc2 if not g & 8 and split == 2 else mc4)
    assert splits == {1, 2, 4}
    assert rules.gemm(256, 2048, 32, 1, 0, 74, 37) & 7 == 4          # without that duty a few tiles still split


def test_raw_q_needs_an_output_that_leaves_it_alone(rules):
    """Against a count of shared bytes, over all offsets of small matrices with equal and different strides."""
    rows = 3
    for stride, width, ostride, owidth in [(16, 4, 16, 4), (16, 8, 16, 8), (16, 6, 16, 12), (16, 16, 16, 16), (16, 4, 32, 8), (24, 8, 16, 8)]:
        q0 = 200
        q = {q0 + r * stride + c for r in range(rows) for c in range(width)}
        for o0 in range(q0 - 120, q0 + 120):
            o = {o0 + r * ostride + c for r in range(rows) for c in range(owidth)}
            got = bool(rules.survives(q0, rows, stride, width, o0, ostride, owidth))
            in_place = (o0, ostride, owidth) == (q0, stride, width)
            if stride == ostride:
                assert got == (in_place or not (q & o)), (stride, width, owidth, o0 - q0)
            else:                                              # different strides: never wrongly allowed, and allowed when the ranges are apart
                assert not (got and q & o) and (got or not (min(o) > max(q) or min(q) > max(o)))


@pytest.mark.parametrize("case", WIDTHS, ids=lambda c: "x".join(map(str, c[:4])))
def test_narrow_gemm_tiles_where_they_measured_faster(case):
    """The width taken is the fastest of the three, within 3 % in single calls and 5.5 % sustained."""
    epi, M, N, K, single, sustained = case
    widths = (256, 224, 192) if N % 256 == 0 else (128, 224, 192)
    w = widths.index(util_routes.linear16_width(M, N, K, epi))
    assert single[w] <= 1.03 * min(single) and sustained[w] <= 1.055 * min(sustained)


def test_no_narrow_gemm_tiles_for_heads_and_few_rows(rules):
    for M, N, ksteps in [(1536, 2048, 32), (3456, 8192, 32), (4096, 2048, 128)]:
        assert rules.width(M, N, ksteps, 1, 0, 0) in (128, 256)      # the head epilogue, whose tiles are whole heads
    assert rules.width(128, 8192, 32, 0, 1, 1) == 128


def test_the_pre_pass_leaves_few_lanes_idle(rules):
    """However few heads there are: a thread block's 2 np pairs per warp are (row, head) pairs of the tensor, up to 3/8 of them (RoPE 1/2)
    and up to the rows that a last thread block lacks; of few heads all of them."""
    for H in range(1, 70):
        for rows in (1, 100, 3000, 40000):
            for in32 in (0, 1):
                for rope in (0, 1):
                    out = (ctypes.c_int * 5)()
                    rules.prep(rows, H, in32, rope, out)
                    np_, few, heads, block_rows, groups = out
                    assert np_ == ((2 if in32 else 4) if rope or rows * H >= 64 * SMS else 1)
                    assert block_rows * heads == 4 * 2 * np_                       # what its four warps can take
                    assert groups * heads >= H and (groups - 1) * heads < H
                    assert 8 * (groups * heads - H) <= (4 if rope else 3) * groups * heads and (not few or groups * heads == H)
