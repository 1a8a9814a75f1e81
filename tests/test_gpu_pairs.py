"""GPU: the explicit pair loop over list orders, lengths and alignments, against FP64 numpy."""
import ctypes as C

import numpy as np
import pytest

from gromos_nb import _lib
from gromos_nb.nonbonded import CRFParameters

pytestmark = pytest.mark.gpu

N, BOX = 600, np.array([3.1, 2.9, 3.3])


def inputs(n_pairs, order, seed=4):
    rng = np.random.default_rng(seed)
    # a jittered lattice: no two atoms nearer than 0.1 nm
    g = np.stack(np.meshgrid(*[np.arange(9)] * 3, indexing="ij"), -1).reshape(-1, 3)[:N]
    x = (g * 0.3 + rng.uniform(-0.1, 0.1, (N, 3))).astype(np.float32)
    i, j = np.triu_indices(N, 1)
    k = rng.permutation(len(i))[:n_pairs]
    if order == "sorted":
        k = np.sort(k)
    elif order == "one":      # one atom's pairs, long runs
        i, j = np.zeros(n_pairs, dtype=int), 1 + np.arange(n_pairs) % (N - 1)
        k = np.arange(n_pairs)
    elif order == "mixed":    # rounds of a few i's
        k = k[np.argsort(i[k] // 3, kind="stable")]
    pairs = np.stack([i[k], j[k]], 1).astype(np.uint32)
    q = rng.normal(0, 0.4, N).astype(np.float32)
    iac = rng.integers(0, 5, N).astype(np.uint32)
    lj = np.abs(rng.normal(1.0, 0.3, (5, 5, 2))) * [2.6e-3, 2.6e-7]
    return x, q, iac, pairs, lj + lj.transpose(1, 0, 2)


def reference(x, q, iac, pairs, lj, crf, box):
    i, j = pairs[:, 0].astype(int), pairs[:, 1].astype(int)
    x, q = x.astype(np.float64), q.astype(np.float64)
    r = x[i] - x[j]
    if box is not None:
        r -= box * np.round(r / box)
    r2 = (r * r).sum(1)
    c = lj[iac[i], iac[j]]
    i6, ir, qq = r2 ** -3.0, r2 ** -0.5, q[i] * q[j] * 138.9354
    fs = (12 * c[:, 1] * i6 - 6 * c[:, 0]) * i6 / r2 + qq * (ir / r2 + crf.crf_cut3i)
    f = np.zeros_like(x)
    np.add.at(f, i, r * fs[:, None])
    np.add.at(f, j, -r * fs[:, None])
    return f, ((c[:, 1] * i6 - c[:, 0]) * i6).sum(), (qq * (ir - crf.crf_2cut3i * r2 - crf.crf_cut)).sum(), \
        r.T @ (r * fs[:, None])


# a round is 32 pairs, a warp's chunk 256, a block's 2048; offsets put pairs and forces 4 bytes off
@pytest.mark.parametrize("n_pairs,order,offset,periodic", [
    (1, "sorted", 0, True), (31, "random", 1, True), (33, "sorted", 0, False), (256, "one", 1, True),
    (257, "mixed", 0, True), (2049, "random", 1, False), (20000, "sorted", 1, True), (60000, "mixed", 0, True),
    (60000, "one", 0, True)])
def test_pair_loop(n_pairs, order, offset, periodic):
    import torch

    x, q, iac, pairs, lj = inputs(n_pairs, order)
    crf = CRFParameters.new(1.4, 1.0, 61.0, 0.0)
    f_ref, lj_ref, crf_ref, v_ref = reference(x, q, iac, pairs, lj, crf, BOX if periodic else None)
    dev = "cuda"

    def shifted(a):  # `offset` 4-byte words into an allocation
        t = torch.zeros(a.size + offset, dtype=torch.int32, device=dev)
        t[offset:] = torch.from_numpy(a.view(np.int32).reshape(-1)).to(dev)
        return t[offset:]

    xd, qd, td, pd, fd = (shifted(a) for a in (x, q, iac, pairs, np.full_like(x, 3.0)))
    ljd = torch.tensor(lj, dtype=torch.float64, device=dev)
    e, v = torch.empty(2, dtype=torch.float64, device=dev), torch.empty(9, dtype=torch.float64, device=dev)
    _lib.check(_lib.lib().gr_lj_crf_innerloop_noalloc(
        xd.data_ptr(), qd.data_ptr(), td.data_ptr(), N, pd.data_ptr(), n_pairs, ljd.data_ptr(), 5,
        BOX.ctypes.data_as(C.c_void_p), 1 if periodic else 0, crf.crf_cut, crf.crf_2cut3i, crf.crf_cut3i,
        fd.data_ptr(), e.data_ptr(), v.data_ptr(), torch.cuda.current_stream().cuda_stream))
    f = fd.cpu().numpy().view(np.float32).reshape(-1, 3).astype(np.float64)
    # a pair's force carries the FP32 rounding of its coordinates (2.7 nm: 1.2e-7 on r >= 0.1 nm, times 13
    # for r^-13), the sums of up to 60,000 pairs on one atom sqrt(n) 6e-8: 2e-5 of the largest covers both
    assert np.abs(f - f_ref).max() <= 2e-5 * np.abs(f_ref).max()
    el, ec = e.tolist()
    assert abs(el - lj_ref) <= 2e-5 * max(abs(lj_ref), abs(crf_ref))
    assert abs(ec - crf_ref) <= 2e-5 * max(abs(lj_ref), abs(crf_ref))
    assert np.abs(v.cpu().numpy().reshape(3, 3) - v_ref).max() <= 2e-5 * np.abs(v_ref).max()


def loop_on_host(x, pairs, c12, box=None, q=None):
    from gromos_nb.nonbonded import lj_crf_innerloop

    n = len(x)
    return lj_crf_innerloop(x, np.zeros(n) if q is None else q, np.zeros(n, dtype=np.uint32), pairs,
                            np.array([[[0.0, c12]]]), CRFParameters.new(1.4, 1.0, 61.0, 0.0), box)


def test_rounding_of_one_pair():
    """Every operation of a pair rounds once, as FP32 division and square root do: the error of r^-14 x
    of separate pairs, whose r^2 is exact, is that of the same operations in numpy."""
    rng = np.random.default_rng(9)
    n = 4000
    d = rng.integers(32, 128, (n, 3)) / 256.0          # 16 bits hold each square, 18 their sum
    x = np.zeros((2 * n, 3), dtype=np.float32)
    x[::2] = d
    pairs = np.arange(2 * n, dtype=np.uint32).reshape(-1, 2)
    f, e_lj, _, _ = loop_on_host(x, pairs, 1e-6)
    r2 = (d * d).sum(1)
    want = 12e-6 * r2 ** -7.0 * d[:, 0]
    s = r2.astype(np.float32)
    i2 = np.float32(1) / s
    i6 = i2 * i2 * i2
    same = np.float32(12) * np.float32(1e-6) * i6 * i6 * i2 * d[:, 0].astype(np.float32)

    def rms(v):
        return np.sqrt((((v - want) / want) ** 2).mean())

    # 1.3: contracted operations round at other places; a reciprocal square root squared gives 2.3
    assert rms(f[::2, 0]) <= 1.3 * rms(same) and rms(f[1::2, 0] * -1.0) <= 1.3 * rms(same)


# 3.38, 3.62, 3.83: 1.5 edges times the rounded reciprocal is below 1.5
@pytest.mark.parametrize("edge,apart,image", [(3.38, 1.5, -0.5), (3.62, 1.5, -0.5), (3.83, 1.5, -0.5), (3.25, 0.5, 0.5),
                                              (3.25, 1.5, -0.5), (3.25, 2.5, 0.5), (2.9, 3.25, 0.25), (3.1, -1.75, 0.25)])
def test_pairs_some_edges_apart(edge, apart, image):
    """A component of `apart` edges is `image` edges: less the nearest whole number, ties to even."""
    edge = np.float32(edge)
    x = np.array([[np.float32(apart) * edge, 0.1, 0.0], [0.0, 0.4, 0.2]], dtype=np.float32)
    assert float(x[0, 0]) == apart * float(edge) or abs(image) != 0.5
    f, _, _, _ = loop_on_host(x, np.array([[0, 1]], dtype=np.uint32), 1e-6, np.array([float(edge)] * 3))
    d = np.array([image * float(edge), -0.3, -0.2])
    assert np.allclose(f[0], 12e-6 * (d @ d) ** -7 * d, rtol=1e-5, atol=0.0) and np.array_equal(f[0], -f[1])


def test_long_lists_leave_no_device_memory_behind():
    """The library's pool keeps blocks for the next call, those of long lists (more than 64 MB) excepted."""
    import torch

    x, q, iac, pairs, lj = inputs(60000, "sorted")
    crf = CRFParameters.new(1.4, 1.0, 61.0, 0.0)
    from gromos_nb.nonbonded import lj_crf_innerloop

    once = lj_crf_innerloop(x, q, iac, pairs, lj, crf, BOX)
    free = torch.cuda.mem_get_info()[0]
    many = lj_crf_innerloop(x, q, iac, np.tile(pairs, (150, 1)), lj, crf, BOX)  # 72 MB
    assert torch.cuda.mem_get_info()[0] >= free - (8 << 20)
    # 60,000 and 9,000,000 FP32 additions to the largest sums
    assert np.abs(many[0] - 150.0 * once[0]).max() <= 1e-3 * np.abs(many[0]).max()
    assert many[1] == pytest.approx(150.0 * once[1], rel=1e-5)
