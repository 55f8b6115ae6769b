// Drives the residue form's three kernels (csrc/residue.h) on operand rows read from a file: planes
// of both operands, the GEMM of every modulus, the reconstruction.  Built and run by
// tests/test_gpu_residue_edges.py.
//
// input (little-endian): int32 rows K bits pair, then float64 A[rows][K], B[rows][K]
// output: int32 moduli, error word; float64 A B^T [rows][rows]
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "residue.h"

using namespace gain::split;

namespace {
void check(cudaError_t e, const char* what) {
    if (e == cudaSuccess) return;
    fprintf(stderr, "%s: %s\n", what, cudaGetErrorString(e));
    exit(1);
}
template <class T>
T* device(size_t n) {
    T* p = nullptr;
    check(cudaMalloc((void**)&p, sizeof(T) * n), "cudaMalloc");
    check(cudaMemset(p, 0, sizeof(T) * n), "cudaMemset");
    return p;
}
RowStats stats(int rows) {
    RowStats s;
    memset(&s, 0, sizeof s);
    s.e = device<int>(rows);
    s.nnz = device<int>(rows);
    s.l2 = device<float>(rows);
    s.dn = device<float>(rows);
    return s;
}
}  // namespace

int main(int argc, char** argv) {
    if (argc != 3) return 2;
    FILE* f = fopen(argv[1], "rb");
    int h[4];
    if (!f || fread(h, 4, 4, f) != 4) return 2;
    const int rows = h[0], K = h[1], bits = h[2], kpad = (K + BK - 1) / BK * BK;
    const bool pair = h[3] != 0;
    const int nmod = residue_moduli(bits, kpad), ncols = pair ? 256 : 128, mstep = pair ? 256 : 128;
    if (rows % 256 || nmod < 1) return 2;
    cudaDeviceProp prop;
    check(cudaGetDeviceProperties(&prop, 0), "cudaGetDeviceProperties");
    __nv_bfloat16* planes[2];
    RowStats st[2];
    for (int k = 0; k < 2; ++k) {
        std::vector<double> v((size_t)rows * K);
        if (fread(v.data(), 8, v.size(), f) != v.size()) return 2;
        double* src = device<double>(v.size());
        check(cudaMemcpy(src, v.data(), 8 * v.size(), cudaMemcpyHostToDevice), "cudaMemcpy");
        planes[k] = device<__nv_bfloat16>((size_t)nmod * rows * kpad);
        st[k] = stats(rows);
        SliceArgs a;
        memset(&a, 0, sizeof a);
        a.src = src;
        a.ld_src = K;
        a.nrows = rows;
        a.ncols = K;
        a.kpad = kpad;
        a.slice_stride = (long)rows * kpad;
        a.digits = planes[k];
        a.slices = nmod;
        a.nchunks = 1;
        a.st = st[k];
        a.bits = bits;
        a.tab = k ? nmod : 0;
        check(launch_slice(a, nullptr), "launch_slice");
    }
    fclose(f);
    CUtensorMap ta, tb;
    if (!make_digit_map(&ta, planes[0], kpad, rows, nmod) || !make_digit_map(&tb, planes[1], kpad, rows, nmod, BN / 2))
        return 1;
    std::vector<ResTile> tiles;
    for (int n0 = 0; n0 < rows; n0 += ncols)
        for (int m0 = 0; m0 < rows; m0 += mstep) {
            ResTile t;
            memset(&t, 0, sizeof t);
            t.m0 = m0;
            t.n0 = n0;
            t.nkb = kpad / BK;
            t.ncols = ncols;
            tiles.push_back(t);
        }
    ResTile* d_tiles = device<ResTile>(tiles.size());
    check(cudaMemcpy(d_tiles, tiles.data(), sizeof(ResTile) * tiles.size(), cudaMemcpyHostToDevice), "cudaMemcpy");
    ResGemmArgs g;
    memset(&g, 0, sizeof g);
    g.tiles = d_tiles;
    g.ntiles = (int)tiles.size();
    g.nmod = nmod;
    g.res = device<uint16_t>((size_t)nmod * rows * rows);
    g.plane = (long)rows * rows;
    g.ldr = rows;
    g.err = device<int>(1);
    check(launch_residue_gemm(ta, tb, g, prop.multiProcessorCount, nullptr, pair), "launch_residue_gemm");
    CrtArgs c;
    memset(&c, 0, sizeof c);
    c.res = g.res;
    c.plane = g.plane;
    c.ldr = c.ldo = rows;
    c.nmod = nmod;
    c.bits = bits;
    c.rows = c.cols = c.cols_valid = rows;
    c.A = st[0];
    c.B = st[1];
    c.out = device<double>((size_t)rows * rows);
    crt_constants(&c);
    check(launch_crt(c, nullptr), "launch_crt");
    std::vector<double> out((size_t)rows * rows);
    int head[2] = {nmod, 0};
    check(cudaMemcpy(out.data(), c.out, 8 * out.size(), cudaMemcpyDeviceToHost), "the run");
    check(cudaMemcpy(&head[1], g.err, 4, cudaMemcpyDeviceToHost), "the run");
    f = fopen(argv[2], "wb");
    if (!f) return 2;
    fwrite(head, 4, 2, f);
    fwrite(out.data(), 8, out.size(), f);
    fclose(f);
    return 0;
}
