"""The FP64 kernels at the sizes where their lists and launches change form: K blocks beyond
one list of terms (1024) and off the thread counts, sparse and dense vectors, non-finite
dipole entries, one-block and cluster dot products."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

JMAX = 11


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("nv,JI,JF,zeros", [(600, 1, 2, 0.0), (513, 2, 1, 0.0), (512, 1, 1, 0.75), (31, 3, 4, 0.5),
                                            (1025, 1, 2, 0.3)])
def test_kblock_lists_bit_exact_vs_oracle(built_lib, nv, JI, JF, zeros):
    import torch
    import gainls
    import oracle
    import synth
    import threej
    bI, bF = synth.make_basis(JI, nv), synth.make_basis(JF, nv)
    rng = np.random.default_rng(nv)
    vec = rng.standard_normal(bI.dimen)
    vec[rng.random(bI.dimen) < zeros] = 0.0
    dip = synth.make_dipole(nv)
    if zeros:     # a skipped lower function's dipole entries are never read into the sum
        lost = np.setdiff1d(np.arange(nv), bI.vib[vec != 0.0])
        dip[:, lost, :] = np.inf
        dip[0, 0, 0] = np.nan
    tj = threej.threej_table(JMAX)
    s, e = 1, nv - 1
    piece = np.ascontiguousarray(dip[:, :, s:e]).reshape(-1)
    ref = np.full(bF.dimen, -7.0)
    d = [_dev(x) for x in (bI.tau, bF.tau, bI.vib, bF.vib, bI.kblock, piece, vec, tj)]
    out = torch.full((bF.dimen,), -7.0, dtype=torch.float64, device="cuda")
    for kF in range(JF + 1):
        if kF - 1 > JI:
            continue
        args = (int(bF.kblock[kF]), bI.dimen, JI, JF, kF)
        at = (int(bF.kstart[kF]), int(bI.kstart[max(kF - 1, 0)]), s, e, e - s)
        oracle.hls_kblock(*args, bI.tau, bF.tau, bI.vib, bF.vib, *at, bI.kblock, piece, nv, vec, tj, JMAX, ref, oracle.REF)
        gainls.hls_kblock(*args, d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(), d[3].data_ptr(), *at,
                          int(bF.kblock[kF]), d[4].data_ptr(), d[5].data_ptr(), d[6].data_ptr(), d[7].data_ptr(),
                          out.data_ptr(), JMAX, nv)
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    assert np.array_equal(np.isnan(got), np.isnan(ref))
    keep = ~np.isnan(ref)
    assert np.array_equal(got[keep].view(np.uint64), ref[keep].view(np.uint64))


@pytest.mark.parametrize("n", [0, 1, 1024, 4095, 4096, 4097, 8192, 8193, 32768 + 5, 1000003])
def test_dot_one_block_and_cluster(built_lib, n):
    """Any n against the double-double sum, within the bound of an FP64 sum of n products; the
    same inputs give the same bits again, on another stream too."""
    import torch
    import gainls
    import oracle
    rng = np.random.default_rng(n)
    x, y = rng.standard_normal(max(n, 1)), rng.standard_normal(max(n, 1))
    dx, dy = _dev(x), _dev(y)
    res = torch.full((3,), np.nan, dtype=torch.float64, device="cuda")
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    gainls.dot(n, dx.data_ptr(), dy.data_ptr(), res.data_ptr(), torch.cuda.current_stream().cuda_stream)
    gainls.dot(n, dx.data_ptr(), dy.data_ptr(), res[1:].data_ptr(), side.cuda_stream)
    torch.cuda.synchronize()
    got = res.cpu().numpy()
    assert got[0] == got[1] and np.isnan(got[2])
    ref = oracle.dot(x[:n], y[:n], oracle.DD) if n else 0.0
    assert abs(got[0] - ref) <= (n + 1) * 2.0 ** -53 * np.sum(np.abs(x[:n] * y[:n]))


@pytest.mark.parametrize("n", [4097, 5000, 8193])
def test_cluster_dots_back_to_back_on_several_streams(built_lib, n):
    """The shortest sums on the cluster: most of its blocks have no element and reach the exchange of
    the partial sums at once, while other launches keep the chip busy.  Every launch gives the
    bits of the first."""
    import torch
    import gainls
    rng = np.random.default_rng(n)
    dx, dy = _dev(rng.standard_normal(n)), _dev(rng.standard_normal(n))
    res = torch.full((4, 400), np.nan, dtype=torch.float64, device="cuda")
    streams = [torch.cuda.Stream() for _ in range(4)]
    for s in streams:
        s.wait_stream(torch.cuda.current_stream())
    for k in range(res.shape[1]):
        for q, s in enumerate(streams):
            gainls.dot(n, dx.data_ptr(), dy.data_ptr(), res[q, k:].data_ptr(), s.cuda_stream)
    torch.cuda.synchronize()
    got = res.cpu().numpy().view(np.uint64)
    assert np.all(got == got[0, 0]) and np.isfinite(res[0, 0].item())
