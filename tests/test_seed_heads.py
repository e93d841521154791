"""Heads of the LRCS scan's hashed table, from the engine's own size functions (host code):
at every length a scan CTA leaves an SM as many CTAs as with 4096 heads, so a longer
table never costs a resident CTA, and a CDS that fits with 4096 heads still fits."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
PKG = ROOT / "protein_encoding_v2_nsga-iii_b200"
SRC = r"""
#include <cstdio>
#include "pe_internal.h"
int main() {
    for (int q = 0; q < 2; q++)
        for (int nt = 64; nt <= 256; nt *= 2)
            for (int n = 9; n <= 48000; n += 3) {
                pe::Shape s{};
                s.L = n / 3, s.m = 2, s.n = n, s.W = (n + 31) / 32, s.Wp = (s.W + 2) & ~1, s.sl_kind = PE_SL_LRCS;
                pe::Shape b = s;
                b.sl_method = 1;  // the band tables alone
                const int ctas = pe::sl_scan_ctas(s, nt, q), heads = pe::sl_seed_heads(s, nt, q, ctas);
                printf("%d %d %d %d %zu %zu %d\n", q, nt, n, heads, pe::sl_scan_smem_bytes(s, nt, heads),
                       pe::sl_scan_smem_bytes(b, nt, heads), pe::sl_seed_heads(s, nt, q, 1));
            }
}
"""
SM, SYSTEM, STATIC = 228 * 1024, 1024, {0: 16, 1: 4128}


@pytest.fixture(scope="module")
def sizes(pe, tmp_path_factory):
    pe.lib()
    d = tmp_path_factory.mktemp("heads")
    (d / "t.cpp").write_text(SRC)
    cuda = next(p for p in (Path("/usr/local/cuda/include"), Path("/usr/local/cuda/targets/x86_64-linux/include"))
                if (p / "cuda_runtime.h").exists())
    lib = PKG / "lib"
    subprocess.run(["g++", "-std=c++17", "-I", str(PKG / "csrc"), "-I", str(cuda), str(d / "t.cpp"), "-o", str(d / "t"),
                    "-L", str(lib), "-lpe_nsga3", f"-Wl,-rpath,{lib}"], check=True)
    out = subprocess.run([str(d / "t")], check=True, capture_output=True, text=True).stdout
    return [tuple(int(x) for x in line.split()) for line in out.splitlines()]


def test_more_heads_never_cost_a_cta(sizes):
    per_sm = lambda b, q: SM // (((b + STATIC[q] + 127) // 128) * 128 + SYSTEM)
    assert len(sizes) > 90000
    seen = set()
    for q, nt, n, heads, got, band, alone in sizes:
        # the bytes with 4096 heads: the rest of the CTA and its nodes, or the band tables
        base = got - (4 * heads + ((4 * n + 15) & ~15))      # exact where the seed table decides the size
        least = max(band, base + 4 * 4096 + ((4 * n + 15) & ~15))
        if n <= 8192:
            assert heads == max(64, min(4096, 1 << (n - 1).bit_length()))
        else:
            assert heads in (4096, 6144, 8192)
            if per_sm(least, q) == 0:
                continue                        # refused: no CTA fits
            if got > band:
                assert per_sm(got, q) == per_sm(least, q), (q, nt, n, heads)
            seen.add(heads)
            assert alone >= heads               # beside a member that leaves one CTA an SM
        assert got + STATIC[q] <= 232448
    assert seen == {4096, 6144, 8192}
