"""CPU tests of the rules that pick an attention call's schedule and a GEMM's tile shape (kiln_b200/csrc/routes.h, plain C++)."""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "kiln_b200", "csrc")
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


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("routes")
    src = d / "routes.cpp"
    src.write_text('#include "routes.h"\n'
                   'extern "C" int route(int B, int Tq, int Tk, int H, int sms, int keys, int room) { return kb::attn_route(B, Tq, Tk, H, sms, keys, room); }\n'
                   'extern "C" int gemm(int M, int N, int ksteps, int n_seg, int any, int mc2, int mc4) {\n'
                   '    const int mc[3] = {0, mc2, mc4}; const kb::GemmShape g = kb::gemm_shape(M, N, ksteps, n_seg, any, 148, mc); return g.pair * 8 + g.split; }\n'
                   'extern "C" int width(int M, int N, int ksteps, int any) {\n'
                   '    const int mc[3] = {0, 74, 37}; return kb::gemm_shape(M, N, ksteps, 1, false, 148, mc, any).width; }\n'
                   'extern "C" void prep(int rows, int H, int in32, int rope, int* out) {\n'
                   '    const kb::PrepLayout l = kb::prep_layout((long long)rows * H, H, in32, rope, 148);\n'
                   '    out[0] = l.np; out[1] = l.few; out[2] = l.heads; out[3] = l.rows; out[4] = l.groups; }\n'
                   'extern "C" int survives(size_t q, size_t rows, size_t stride, size_t width, size_t o, size_t ostride, size_t owidth) {\n'
                   '    return kb::q_survives_output({(void*)q, rows, stride, width}, {(void*)o, rows, ostride, owidth}); }\n')
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I" + CSRC, "-o", str(d / "routes.so"), str(src)], check=True)
    lib = ctypes.CDLL(str(d / "routes.so"))
    lib.survives.argtypes = [ctypes.c_size_t] * 7
    lib.width.argtypes = [ctypes.c_int] * 4
    return lib


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


def test_narrow_gemm_tiles_where_they_measured_faster(rules):
    """Width of the tiles against device times on a B200 (us): 256, 224 and 192 columns forced in turn."""
    for M, N, ksteps, times in [(1280, 2048, 32, (18.8, 16.4, 14.9)), (1536, 2048, 32, (18.8, 16.6, 15.1)), (1792, 2048, 32, (18.5, 16.6, 21.6)), (2048, 2048, 32, (18.8, 22.8, 22.4)),
                                (2304, 2048, 32, (19.0, 25.3, 22.7)), (2560, 2048, 32, (29.0, 25.5, 22.9)), (3456, 2048, 32, (29.3, 26.5, 30.4)), (4096, 2048, 32, (29.8, 33.7, 31.5)),
                                (1536, 2048, 128, (48.4, 43.2, 40.9)), (3456, 2048, 128, (96.7, 95.0, 112.0)), (4096, 2048, 128, (104.4, 124.7, 119.7)),
                                (512, 8192, 32, (21.1, 18.4, 25.1)), (1024, 8192, 32, (31.3, 28.0, 33.9)), (1536, 8192, 32, (42.8, 40.4, 46.0)), (2304, 8192, 32, (59.2, 63.1, 67.7)),
                                (3456, 8192, 32, (94.9, 92.8, 103.9)), (4096, 8192, 32, (104.0, 106.7, 118.0))]:
        assert rules.width(M, N, ksteps, 1) == (256, 224, 192)[times.index(min(times))], (M, N, ksteps)
        assert rules.width(M, N, ksteps, 0) in (128, 256)            # the head epilogue has no narrow tiles
    assert rules.width(128, 8192, 32, 1) == 128


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
