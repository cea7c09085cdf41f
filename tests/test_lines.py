"""The lines between kernels (csrc/lines.h) at the sizes whose two sides were measured; no GPU is needed."""
import ctypes as C
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "llamd_rs_b200", "csrc")
SOURCE = """
#include "lines.h"
extern "C" {
int experts(long long pairs, int n_expert, long long weights) { return llamd::experts_on_gemm(pairs, n_expert, weights); }
int four_ctas(long long ctas, long long smem) { return llamd::attn_out_four_ctas(ctas, smem); }
int small_tile(int positions, long long ctas) { return llamd::small_tile_by_kv_head(positions, ctas); }
int product(int blocks, int rows, int nseq) { return llamd::product_on_gemm(blocks, rows, nseq); }
}
"""


@pytest.fixture(scope="module")
def lines(tmp_path_factory):
    d = tmp_path_factory.mktemp("lines")
    (d / "l.cpp").write_text(SOURCE)
    subprocess.check_call(["g++", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(d / "l.cpp"), "-o", str(d / "l.so")])
    L = C.CDLL(str(d / "l.so"))
    L.experts.argtypes = [C.c_longlong, C.c_int, C.c_longlong]
    L.four_ctas.argtypes = [C.c_longlong, C.c_longlong]
    L.small_tile.argtypes = [C.c_int, C.c_longlong]
    return L


# experts, used per token, width, n_embd; tokens that the matvec is faster for by 2 % and more, tokens that the GEMM is
@pytest.mark.parametrize("n_expert,used,width,embd,matvec,gemm", [
    (8, 2, 1536, 2048, (2, 4, 8), (12, 16, 24)), (8, 2, 3072, 4096, (4, 6), (10, 12, 32)), (16, 2, 1536, 4096, (8, 12, 14), (16, 20, 64)),
    (16, 2, 256, 2048, (8, 16, 18), (36, 56, 64)), (32, 4, 768, 2048, (8, 14, 16), (20, 24, 32)), (64, 8, 768, 2048, (8, 14), (18, 20, 32)),
    (64, 6, 1536, 2048, (10, 16, 18), (24, 28, 64)), (60, 4, 1536, 2048, (12, 20, 24), (32, 36, 64)), (64, 4, 256, 2048, (14, 32, 36), (48, 56, 64)),
    (128, 8, 768, 2048, (8, 24), (32, 36, 64)), (128, 8, 256, 2048, (14, 28, 32), (44, 48, 64)), (128, 8, 512, 1024, (14, 28, 32), (44, 48, 64)),
    (256, 8, 512, 2048, (32, 48, 56), (70,)), (512, 10, 512, 2048, (26, 51, 64), (120,))])
def test_experts_change_over_by_pairs_per_expert(lines, n_expert, used, width, embd, matvec, gemm):
    assert not any(lines.experts(n * used, n_expert, width * embd) for n in matvec)
    assert all(lines.experts(n * used, n_expert, width * embd) for n in gemm)


def _values_smem(positions):
    return 4 * (8 * ((positions + 3) & ~3) + 2 * 128 * 32)  # eight rows of scores, two tiles of values


def test_four_attention_ctas_only_where_they_are_there(lines):
    for n in (37, 96, 128, 256):  # sequences, or tokens of a small tile: 16 CTAs each
        assert all(lines.four_ctas(16 * n, _values_smem(p)) for p in (40, 288, 700, 768)), n
        assert not any(lines.four_ctas(16 * n, _values_smem(p)) for p in (769, 837, 1000, 1500, 2500, 4000)), n
    assert not any(lines.four_ctas(16 * n, _values_smem(288)) for n in (4, 9, 32))


def test_small_tiles_by_kv_head_behind_long_contexts(lines):
    assert all(lines.small_tile(p, 16 * n) for p in (40, 1000, 4352) for n in (2, 9, 37, 56))
    for p in (4356, 4800, 5376):
        assert all(lines.small_tile(p, 16 * n) for n in (2, 4, 9))
        assert not any(lines.small_tile(p, 16 * n) for n in (14, 19, 24, 37, 56))
    assert not any(lines.small_tile(5380, 16 * n) for n in (2, 9, 56))


# rows x blocks, sequences that the matvec is faster for (or as fast), sequences that the GEMM is
@pytest.mark.parametrize("rows,blocks,matvec,gemm", [
    (2048, 8, (1, 2), (3, 4, 8)), (151936, 8, (1, 2), (3, 4, 8)), (5120, 1, (2,), (3, 8)), (512, 16, (2, 3, 5), ()), (1024, 16, (2, 3), (6, 8)),
    (2048, 16, (2,), (4, 6, 8)), (1024, 12, (3, 4), (6, 8)), (20000, 16, (2,), (3, 8)), (512, 20, (3, 4, 6, 8), ()), (1024, 20, (3, 5), (8,)),
    (3072, 20, (2, 3, 4), (5, 6, 8)), (512, 24, (2, 3, 4, 5), ()), (2048, 24, (2,), (3, 4, 8)), (3072, 24, (2, 3), (4, 6, 8)),
    (10000, 24, (2,), (3, 4, 8)), (5120, 25, (2, 3, 8), ())])
def test_products_of_several_sequences(lines, rows, blocks, matvec, gemm):
    assert not any(lines.product(blocks, rows, n) for n in matvec)
    assert all(lines.product(blocks, rows, n) for n in gemm)
