"""The separable 3D vote of sparse fields against FP64: receivers that only far
voters reach keep the accuracy of a near voter's, relative to the Gaussian
weight that the voters have there.

Tolerance, in units of sum over voters of scale * (c1 + c2): the tables give
1.5e-7.  A term of a vote is a product of three axis weights, a moment (up to
8 operations) and two coefficients, added up along some 10 further roundings;
the terms' magnitudes come to some 20 times the vote.  20 sqrt(23) 2^-24 =
5.7e-6; with the tables', 6e-6."""
import numpy as np
import pytest

from oracle import oracle as O
from test_gpu_vote3_sep import THREADS, WGT, kernels_of

pytestmark = pytest.mark.gpu

TOL = 6e-6


def sparse_field(shape, seed, count, kind):
    rng = np.random.default_rng(seed)
    T = np.zeros(shape + (3, 3), np.float32)
    at = np.stack([rng.integers(0, s, count) for s in shape], 1)
    for p in at:
        q = rng.normal(size=3)
        q /= np.linalg.norm(q)
        M = {"stick": np.outer(q, q), "plate": np.eye(3) - np.outer(q, q), "mix": np.eye(3) + 2 * np.outer(q, q)}[kind]
        T[tuple(p)] = M * 10.0 ** rng.uniform(-3, 3)
    return T, at


@pytest.mark.parametrize("shape,sigma,sigma2,w,kind,opts", [
    ((96, 96, 96), 2.2, 0.0, 0, "stick", {}),
    ((96, 96, 96), 4.0, 0.0, 0, "stick", {}),
    ((96, 96, 96), 4.0, 0.0, 0, "plate", {}),
    ((64, 96, 96), 6.0, 0.0, 0, "mix", {"ball": True}),
    ((64, 96, 96), 6.8, 0.0, 41, "stick", {}),
    ((64, 96, 96), 2.5, 0.0, 25, "plate", {}),             # a window of five sigma
    ((64, 96, 96), 4.0, 1.0, 0, "stick", {}),              # the second Gaussian far narrower
    ((64, 96, 96), 2.0, 5.0, 0, "mix", {}),                # and the first
    ((64, 96, 96), 3.0, 3.0, 0, "plate", {}),
])
def test_far_receivers_keep_their_accuracy(shape, sigma, sigma2, w, kind, opts):
    import torch
    import tiralib_gb300 as tv
    hw = (w or 2 * int(np.float32(3.0) * np.float32(max(sigma, sigma2))) + 1) // 2
    T, at = sparse_field(shape, 7, 6, kind)
    (out, _, _), names = kernels_of(lambda: tv.vote3(torch.from_numpy(T).cuda(), sigma, sigma2, w=w, parity=False,
                                                     out_layout="sym6", **opts))
    assert "k_sep_xy" in names
    # receivers of every voter: the window's corners, edges and faces, and others at random
    rng = np.random.default_rng(8)
    g = np.array([-hw, -hw // 2, 0, hw // 2, hw])
    off = np.concatenate([np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3),
                          rng.integers(-hw, hw + 1, (200, 3))])
    rec = np.unique((at[:, None] + off[None]).reshape(-1, 3), axis=0)
    rec = rec[((rec >= 0) & (rec < np.array(shape))).all(1)]
    idx = (rec[:, 0] * shape[1] + rec[:, 1]) * shape[2] + rec[:, 2]
    ref = O.tensorvote3_f64(T, sigma, sigma2, 2 * hw + 1, 1, receivers=idx, threads=THREADS, **opts).reshape(-1, 6)[idx]
    got = out.cpu().numpy().reshape(-1, 6)[idx].astype(np.float64)
    weight = np.zeros(len(rec))
    for p in at:
        d = rec - p
        s = (d ** 2).sum(1).astype(float)
        c = np.exp(-s / sigma ** 2) + (np.exp(-s / sigma2 ** 2) if sigma2 else 0.0)
        sn = tv.sticknorm3(sigma, sigma2, 1) if kind != "plate" else 1.0
        size = np.linalg.norm(T[tuple(p)]) * max(1.0, 1.0 / sn)
        weight += np.where((np.abs(d) <= hw).all(1), size * c, 0.0)
    err = np.sqrt((WGT * (got - ref) ** 2).sum(1))
    assert (got[weight == 0.0] == 0.0).all()
    assert (err <= TOL * weight).all()


def test_far_receivers_of_the_anisotropic_vote():
    """ATV: the same sums with one Gaussian; a lone stick at every offset of
    its window."""
    import torch
    import tiralib_gb300 as tv
    n, hw, sigma = 64, 12, 4.0
    q = np.array([0.3, -0.5, 0.8])
    q /= np.linalg.norm(q)
    T = np.zeros((n, n, n, 3, 3), np.float32)
    T[32, 32, 32] = np.outer(q, q)
    (out, _, _), names = kernels_of(lambda: tv.vote3(torch.from_numpy(T).cuda(), sigma, w=25, is_atv=True,
                                                     out_layout="sym6", parity=False))
    assert "k_sep_xy" in names
    g = np.arange(-hw, hw + 1)
    o = np.stack(np.meshgrid(g, g, g, indexing="ij")[::-1], -1).astype(float)     # x, y, z of receiver - voter
    s = (o ** 2).sum(-1)
    lam, vec = np.linalg.eigh(T[32, 32, 32].astype(np.float64))
    d = o / np.sqrt(np.where(s > 0, s, 1.0))[..., None]
    I = np.eye(3)
    H = np.zeros(o.shape[:-1] + (3, 3))
    terms = [(lam[2] - lam[1], np.outer(vec[:, 2], vec[:, 2]), 3),
             (lam[1] - lam[0], np.outer(vec[:, 2], vec[:, 2]) + np.outer(vec[:, 1], vec[:, 1]), 4), (lam[0], I, 5)]
    for scale, M, k in terms:
        v = d @ M
        vv = (v * d).sum(-1)
        H += scale * (M - (M * vv[..., None, None] + 2 * v[..., :, None] * v[..., None, :]) / k)
    R = I - 2 * d[..., :, None] * d[..., None, :]
    ref = np.exp(-s / sigma ** 2)[..., None, None] * (R @ H @ R)
    iu = ([0, 0, 0, 1, 1, 2], [0, 1, 2, 1, 2, 2])
    got = out.cpu().numpy()[32 - hw:32 + hw + 1, 32 - hw:32 + hw + 1, 32 - hw:32 + hw + 1].astype(np.float64)
    err = np.sqrt((WGT * (got - ref[..., iu[0], iu[1]]) ** 2).sum(-1))
    assert (err <= TOL * np.exp(-s / sigma ** 2)).all()
