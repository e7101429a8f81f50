"""Parts of the library that whole solves reach only indirectly, through a small
program linked against libtdz.so (tests/native/gpu_parts_check.cpp): the
eigenvector transforms that read and write natural-order FP64 vectors, with the
fused norm of the latter, at the edges of their tiles, and the 2D soft-core term
without its table."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.fixture(scope="module")
def parts(cuda, tmp_path_factory):
    from tdsez_gb300 import build
    exe, pkg = str(tmp_path_factory.mktemp("parts") / "gpu_parts_check"), os.path.join(ROOT, "tdsez_gb300")
    subprocess.run([build.nvcc(), "-O2", "-std=c++17", "-I", os.path.join(pkg, "csrc"), "-I",
                    os.path.join(ROOT, "include"), os.path.join(HERE, "native", "gpu_parts_check.cpp"), "-o", exe,
                    "-L", pkg, "-ltdz", "-Xlinker", "-rpath=" + pkg, "-lcudart"], check=True)

    def run(line):
        r = subprocess.run([exe], input=line + "\n", capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr
        return r.stdout.split()
    return run


@pytest.mark.gpu
@pytest.mark.parametrize("K,N,planes,R", [
    (1, 1, 1, 1),          # one row pair of one tile
    (16, 16, 1, 64),       # one full tile, one chunk, one column group
    (17, 17, 1, 65),       # one past each
    (40, 5, 3, 21),        # fewer columns than a group
    (163, 163, 2, 163),    # the benchmark's axis, partial last tile
    (176, 176, 1, 300),    # the largest resident matrix
    (250, 112, 2, 65),     # few stages
    (33, 49, 310, 64),     # two tiles per CTA with a remainder, odd column groups
])
@pytest.mark.parametrize("way", ["from64", "to64"])
def test_fp64_ends(parts, way, K, N, planes, R):
    err, norm, bad = parts(f"{way} {K} {N} {planes} {R}")
    assert int(bad) == 0
    # 24-bit operands in three slices and an FP32 sum of K products, as in the planar
    # form: (K + 4) 2^-24 of sum |x b|, below 6 times the largest result
    assert float(err) <= 6 * (K + 4) * 2.0 ** -24
    # FP32 sums of at most 48 squares of a row's half, FP64 beyond
    assert float(norm) <= 48 * 2.0 ** -24


@pytest.mark.gpu
@pytest.mark.parametrize("p,nq,nx,ny", [(2, 3, 1, 1), (2, 3, 40, 9), (3, 4, 33, 12), (4, 5, 30, 31), (5, 6, 28, 7),
                                        (3, 6, 17, 20), (5, 2, 19, 11)])
@pytest.mark.parametrize("prec", [0, 1])
def test_quad2_without_table(parts, p, nq, nx, ny, prec):
    err, held = parts(f"quad2 {p} {nq} {nx} {ny} {prec}")
    # the table of the applied precision only; none past the limit
    assert held == ("1000" if prec else "0100")
    # both forms within the bars of the apply parity tests
    assert float(err) < (2e-12 if prec else 2e-6)
