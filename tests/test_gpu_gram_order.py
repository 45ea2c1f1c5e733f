"""GPU: the order of summation of the narrow FP64 Gram products (dense_fp64.cu), bit for bit, and rotations of few
rows.

The signs of the eigensolver's vectors turn on the last bits of these products, which rest on an FP64 matrix
instruction adding its four products one after the other like four FMAs.  The chains, their tree and the
sum over blocks are restated in C with fma()."""
import ctypes as C
import subprocess

import numpy as np
import pytest

import dft_b200

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include <math.h>
static double tree(double *c) {  /* 32 values, butterfly */
    for (int o = 16; o > 0; o >>= 1)
        for (int l = 0; l < o; ++l) c[l] = c[l] + c[l + o];
    return c[0];
}
/* points dealt to nblk blocks of 32 chains: chain (b, l) takes 32 b + l + 32 m nblk */
double lanes(const double *a, const double *b, long n, long nblk, double scale) {
    double total = 0.0, group = 0.0;
    for (long k = 0; k < nblk; ++k) {
        double c[32];
        for (int l = 0; l < 32; ++l) {
            c[l] = 0.0;
            for (long p = 32 * k + l; p < n; p += 32 * nblk) c[l] = fma(a[p], b[p], c[l]);
        }
        group += tree(c);
        if (k % 16 == 15 || k + 1 == nblk) {  /* 16 blocks in order, then the groups in order */
            total += group;
            group = 0.0;
        }
    }
    return total * scale;
}
/* one chain per chunk of the points; lanes stride the chunks */
double chunks(const double *a, const double *b, long n, long chunk, long nch, double scale) {
    double c[32];
    for (int l = 0; l < 32; ++l) {
        c[l] = 0.0;
        for (long k = l; k < nch; k += 32) {
            double s = 0.0;
            for (long p = k * chunk; p < n && p < (k + 1) * chunk; ++p) s = fma(a[p], b[p], s);
            c[l] += s;
        }
    }
    return tree(c) * scale;
}
"""


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    d = tmp_path_factory.mktemp("gram_order")
    (d / "order.c").write_text(SOURCE)
    subprocess.run(["gcc", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-o", str(d / "order.so"), str(d / "order.c"),
                    "-lm"], check=True)
    lib = C.CDLL(str(d / "order.so"))
    P = C.POINTER(C.c_double)
    lib.lanes.argtypes, lib.lanes.restype = [P, P, C.c_long, C.c_long, C.c_double], C.c_double
    lib.chunks.argtypes, lib.chunks.restype = [P, P, C.c_long, C.c_long, C.c_long, C.c_double], C.c_double
    return lib


# both sides of every width at which the order changes, both kernels; even and odd leading dimensions
@pytest.mark.parametrize("dims", [(4, 5, 6), (13, 11, 17), (33, 31, 17), (40, 40, 40)])
@pytest.mark.parametrize("ka,kb", [(1, 1), (8, 8), (5, 12), (9, 5), (20, 4), (24, 12), (33, 8), (64, 4), (33, 9), (64, 16)])
def test_narrow_gram_bits(engine, host, dims, ka, kb):
    torch = pytest.importorskip("torch")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    g = dft_b200.CartesianGrid(*dims, -1.0, 1.0, -1.5, 1.5, -2.0, 2.0)
    N = g.getSize()
    dV = g.getDx() * g.getDy() * g.getDz()
    rng = np.random.default_rng(ka * 100 + kb)
    A, B = rng.standard_normal((ka, N)), rng.standard_normal((kb, N))
    got = engine.gram(g, engine.upload(A), N, ka, engine.upload(B), N, kb)
    rows = 1 if ka <= 8 else 2 if ka <= 16 else 4 if ka <= 32 else 8
    cols = 4 if kb <= 4 else 8 if kb <= 8 else 16
    P = C.POINTER(C.c_double)

    def ptr(x):
        return x.ctypes.data_as(P)

    if rows * cols <= 64:
        nblk = max(1, min(4 * sms, 1024, (N + 255) // 256))

        def one(a, b):
            return host.lanes(ptr(a), ptr(b), N, nblk, dV)
    else:
        nch = max(1, 4 * sms // ((ka + 31) // 32))
        chunk = ((N + nch - 1) // nch + 31) // 32 * 32
        nch = (N + chunk - 1) // chunk
        chunk = (N + nch - 1) // nch

        def one(a, b):
            return host.chunks(ptr(a), ptr(b), N, chunk, nch, dV)

    # every row tile and column tile, first and last of each
    for i in sorted({0, ka // 2, ka - 1, min(7, ka - 1), min(8, ka - 1)}):
        for j in sorted({0, kb // 2, kb - 1, min(7, kb - 1)}):
            assert got[i, j] == one(A[i], B[j]), (i, j)


# few rows of the block that is rotated: a warp then takes more points (ragged ends of 64)
@pytest.mark.parametrize("dims", [(2, 2, 2), (5, 7, 3), (8, 8, 8), (33, 31, 17)])
@pytest.mark.parametrize("k,m", [(1, 8), (2, 5), (3, 3), (3, 9), (4, 4)])
def test_rotation_of_few_rows(engine, dims, k, m):
    g = dft_b200.CartesianGrid(*dims, -1.0, 1.0, -1.5, 1.5, -2.0, 2.0)
    N = g.getSize()
    rng = np.random.default_rng(k * 100 + m)
    V, Y = rng.standard_normal((k, N)), rng.standard_normal((k, m))
    X = engine.upload(np.full((m, N), 7.0))
    engine.rotate(g, engine.upload(V), N, k, Y, X, N)
    # k products and sums in any order: |error| <= (k + 2) eps sum |y||v|
    bound = (k + 2) * 2.0 ** -53 * (np.abs(Y).T @ np.abs(V))
    assert np.all(np.abs(X.to_host((m, N)) - Y.T @ V) <= 2 * bound)
