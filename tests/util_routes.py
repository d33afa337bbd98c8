"""The rules of kiln_b200/csrc/routes.h (plain C++) as Python functions, for a GPU of 148 SMs: the CPU tests hold them to measurements, GPU tests
assert with them that a case takes the route it is there for."""
import ctypes
import functools
import os
import subprocess
import tempfile

SMS = 148
CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "kiln_b200", "csrc")
SOURCE = r"""
#include "routes.h"
extern "C" {
int route(int B, int Tq, int Tk, int H, int sms, int keys, int room) { return kb::attn_route(B, Tq, Tk, H, sms, keys, room); }
int gemm(int M, int N, int ksteps, int n_seg, int any, int mc2, int mc4) {
    const int mc[3] = {0, mc2, mc4};
    const kb::GemmShape g = kb::gemm_shape(M, N, ksteps, n_seg, any, 148, mc);
    return g.pair * 8 + g.split;
}
int width(int M, int N, int ksteps, int any_n_seg, int any, int gelu) {
    const int mc[3] = {0, 74, 37};
    return kb::gemm_shape(M, N, ksteps, 1, any_n_seg, 148, mc, any, gelu).width;
}
void prep(int rows, int H, int in32, int rope, int* out) {
    const kb::PrepLayout l = kb::prep_layout((long long)rows * H, H, in32, rope, 148);
    out[0] = l.np; out[1] = l.few; out[2] = l.heads; out[3] = l.rows; out[4] = l.groups;
}
int q_per(int B, int Tq, int Tk, int H) {
    int qsplit, q_per;
    kb::bwd_qsplit(B, Tq, Tk, H, 148, &qsplit, &q_per);
    return q_per;
}
int survives(size_t q, size_t rows, size_t stride, size_t width, size_t o, size_t ostride, size_t owidth) {
    return kb::q_survives_output({(void*)q, rows, stride, width}, {(void*)o, rows, ostride, owidth});
}
}
"""


@functools.lru_cache(None)
def rules():
    with tempfile.TemporaryDirectory() as d:
        src, out = os.path.join(d, "routes.cpp"), os.path.join(d, "routes.so")
        with open(src, "w") as f:
            f.write(SOURCE)
        subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I" + CSRC, "-o", out, src], check=True)
        lib = ctypes.CDLL(out)
    lib.survives.argtypes = [ctypes.c_size_t] * 7
    return lib


def linear16_width(M, N, K, epi):
    """Columns of a tile of one linear16 call with epilogue "F32", "F16", "GELU16" or "RESID"."""
    return rules().width(M, N, K // 64, epi == "F16" and N % 128 == 0, 1, epi == "GELU16")


def bwd_q_per(B, Tq, Tk, H):
    """Query blocks that a thread block of the dK/dV role streams at most."""
    return rules().q_per(B, Tq, Tk, H)
