"""Subtomogram averaging on the GPU against the FP64 restatement of BH_average3d's loop."""
import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _case(seed, n=40, k=10, nw=36, n_wedges=2):
    from emclarity_b200 import api, synthetic
    rng = np.random.default_rng(seed)
    ref = synthetic.blob_reference(rng, n)
    parts, rots, shifts, weights, halves, widx = [], [], [], [], [], []
    for i in range(k):
        R = api.define_matrix(synthetic.random_euler(rng), "inv")
        t = rng.uniform(-1.5, 1.5, 3)
        # the window holds the reference rotated forward by R and shifted; the average rotates it back
        vol = O.rotate(ref, R.T, t, "forward", interp=2) + 0.3 * rng.standard_normal((n, n, n))
        parts.append(vol.astype(np.float32))
        rots.append(R)
        shifts.append(t)
        weights.append(rng.uniform(0.5, 1.0))
        halves.append(1 + (i % 2))
        widx.append(i % n_wedges)
    mask = synthetic.soft_sphere_mask(n, 0.35 * n)
    wedges = [np.abs(rng.standard_normal((nw, nw, nw))).astype(np.float32) for _ in range(n_wedges)]
    return dict(parts=np.array(parts), rots=np.array(rots), shifts=np.array(shifts, np.float32),
                weights=np.array(weights, np.float32), halves=np.array(halves), widx=np.array(widx),
                mask=mask, wedges=np.array(wedges), ref=ref)


def _run_gpu(c, symmetry="C1", batch=0, wedges=True):
    from emclarity_b200 import api
    nw = c["wedges"].shape[-1] if wedges else 0
    avg = api.Average(torch.from_numpy(c["mask"]).cuda(), symmetry=symmetry, wedge_box=nw, batch=batch)
    kept = avg.add(torch.from_numpy(c["parts"]).cuda(), c["rots"], c["halves"], shifts=c["shifts"],
                   weights=c["weights"], wedges=torch.from_numpy(c["wedges"]).cuda() if wedges else None,
                   wedge_index=c["widx"] if wedges else None)
    out = {h: avg.result(h) for h in (1, 2)}
    avg.close()
    return out, kept


def _run_oracle(c, symmetry=None, wedges=True):
    return O.average_np(list(c["parts"]), c["mask"], list(c["rots"]), c["halves"], shifts=c["shifts"],
                        weights=c["weights"], wedges=list(c["wedges"]) if wedges else None,
                        wedge_index=c["widx"] if wedges else None, symmetry=symmetry)


@pytest.mark.parametrize("symmetry", ["C1", "C3"])
def test_average_matches_oracle(built_lib, cuda, symmetry):
    from emclarity_b200 import api
    c = _case(11)
    g, kept = _run_gpu(c, symmetry)
    o, kept_o = _run_oracle(c, O.symmetry_matrices_np(symmetry))
    assert kept.all() and kept_o.all()
    for h in (1, 2):
        avg, wsum, cnt = g[h]
        oa, ow, oc = o[h]
        assert cnt == oc == 5
        a = avg.cpu().numpy()
        assert np.abs(a - oa).max() <= 2e-5 * np.abs(oa).max(), np.abs(a - oa).max()
        w = wsum.cpu().numpy()
        assert np.abs(w - ow).max() <= 2e-5 * np.abs(ow).max()


def test_average_recovers_the_reference(built_lib, cuda):
    """Aligned, noisy copies average back to (a masked, normalised) reference."""
    c = _case(12, k=16)
    g, _ = _run_gpu(c, wedges=False)
    a = (g[1][0].cpu().numpy() + g[2][0].cpu().numpy()) / 2
    r = c["ref"] * c["mask"]
    cc = np.sum((a - a.mean()) * (r - r.mean())) / np.sqrt(np.sum((a - a.mean()) ** 2) * np.sum((r - r.mean()) ** 2))
    assert cc > 0.9, cc


def test_batches_give_identical_sums(built_lib, cuda):
    """Particles are added in order whatever the batch split: bit-identical results."""
    c = _case(13, k=7)
    a, _ = _run_gpu(c, batch=0)
    b, _ = _run_gpu(c, batch=3)
    for h in (1, 2):
        assert torch.equal(a[h][0], b[h][0]) and torch.equal(a[h][1], b[h][1]) and a[h][2] == b[h][2]


def test_non_finite_particle_is_dropped(built_lib, cuda):
    c = _case(14, k=4)
    c["parts"][2, 20, 20, 20] = np.nan
    g, kept = _run_gpu(c)
    o, kept_o = _run_oracle(c)
    assert list(kept) == list(kept_o) == [True, True, False, True]
    for h in (1, 2):
        assert g[h][2] == o[h][2]
        assert np.isfinite(g[h][0].cpu().numpy()).all()


def test_empty_half_set_is_nan_and_bad_arguments(built_lib, cuda):
    from emclarity_b200 import EmcError, api
    c = _case(15, k=2)
    c["halves"][:] = 1
    g, _ = _run_gpu(c, wedges=False)
    assert g[2][2] == 0 and torch.isnan(g[2][0]).all()
    avg = api.Average(torch.from_numpy(c["mask"]).cuda())
    with pytest.raises(EmcError):
        avg.add(torch.from_numpy(c["parts"]).cuda(), c["rots"], [1, 3])
    with pytest.raises(EmcError):
        avg.result(0)
    with pytest.raises(EmcError):
        api.Average(torch.zeros(8, 8, 8, device="cuda"))  # no voxel above the threshold
    avg.close()


@pytest.mark.parametrize("n,nw", [(33, 17), (34, 9), (16, 16), (50, 48)])
def test_brick_edges_and_wide_matrices(built_lib, cuda, n, nw):
    """Edges that end inside a brick and each copy width (odd, even and multiple-of-four boxes), and
    matrices that scale by 2.5 (their source box is larger than the staging, so the samples come from
    global memory) beside rotations; same tolerance as the other boxes."""
    c = _case(20 + n, n=n, k=4, nw=nw)
    c["rots"][1] = 2.5 * c["rots"][1]
    c["shifts"][2] = (40.0 * n, 0.0, 0.0)  # the window of particle 2 lies outside: no finite rms, dropped
    g, kept = _run_gpu(c)
    with np.errstate(invalid="ignore", divide="ignore"):
        o, kept_o = _run_oracle(c)
    assert list(kept) == list(kept_o) == [True, True, False, True]
    for h in (1, 2):
        assert g[h][2] == o[h][2]
        for k in (0, 1):
            a, b = g[h][k].cpu().numpy(), o[h][k]
            assert np.abs(a - b).max() <= 2e-5 * np.abs(b).max(), (h, k)


@pytest.mark.parametrize("windows", [1, 12])
def test_cancelling_matrices_on_thin_bricks(built_lib, cuda, windows):
    """A box one voxel longer than whole bricks, with matrices whose entries are huge and cancel (or are
    cancelled by the shift) at its far corner: the sums in different orders differ by whole voxels there,
    so those samples do not come from the staged box.  The window's samples lie beyond it almost
    everywhere; with one window (too few CTAs to stage) and with several equal ones; against a float32 restatement of the sampling in the kernel's order (FP32 products are
    exact in float64, so one rounding each), whose coordinates must agree bit for bit."""
    from emclarity_b200 import api
    n, c = 17, 8
    rng = np.random.default_rng(17)
    vol = rng.standard_normal((n, n, n)).astype(np.float32)
    cases = [(np.array([[1e7 + 3, -1e7, 0.3], [0, 1, 0], [0, 0, 1]]), (0, 0, 0)),
             (np.array([[1, 0, 0], [0.25, 3e6, -3e6], [0, 0, 1]]), (0, -1.5, 0)),
             (np.array([[1, 0, 0], [0, 1, 0], [0.3, 0.3, 2e6]]), (0, 0, -1.6e7)),
             (np.eye(3), (0.5, 0.25, -0.75))]
    mask = torch.ones((n, n, n), device="cuda")

    def fma(a, b, d):  # one rounding: the product of two floats is exact in 64 bits, the sum nearly so
        return (a.astype(np.float64) * b.astype(np.float64) + d.astype(np.float64)).astype(np.float32)

    z, y, x = np.meshgrid(*[np.arange(n, dtype=np.float32) - c] * 3, indexing="ij")
    for m, t in cases:
        m32, t32 = m.astype(np.float32), np.asarray(t, np.float32)
        s = []
        for i in range(3):
            v = fma(m32[i, 0:1], x, fma(m32[i, 1:2], y, (m32[i, 2] * z).astype(np.float32)))
            s.append(((v + t32[i]).astype(np.float32) + np.float32(c)).astype(np.float64))
        want = np.zeros((n, n, n))
        for k in range(8):
            o = (k & 1, (k >> 1) & 1, k >> 2)
            w, ok, idx = 1.0, True, []
            for a, oi in zip(s, o):
                b = np.floor(a)
                f = a - b
                w = w * (f if oi else 1 - f)
                ok = ok & (b + oi >= 0) & (b + oi < n)
                idx.append(np.clip(b + oi, 0, n - 1).astype(int))
            want += np.where(ok, w * vol[idx[2], idx[1], idx[0]], 0.0)
        av = api.Average(mask)
        kept = av.add(torch.from_numpy(np.stack([vol] * windows)).cuda(), [m] * windows, [1] * windows,
                      shifts=[t] * windows)
        assert kept.all()
        got = av.result(1)[0].cpu().numpy()
        av.close()
        want = (want - want.mean()) / want.std()
        assert np.abs(got - want).max() <= 2e-5 * np.abs(want).max()


@pytest.mark.parametrize("n,nw", [(17, 16), (33, 31), (40, 34)])
def test_one_window_at_a_time_matches_a_batch(built_lib, cuda, n, nw):
    """Few CTAs (one window) sample global memory in thin bricks, a batch stages boxes: the rotated values
    are the same, the FP64 statistics differ by their order, so the sums differ by a rounding of each
    window's mean, rms and quotient."""
    c = _case(n, n=n, k=24, nw=nw)
    from emclarity_b200 import api
    sums = []
    for step in (24, 1):
        av = api.Average(torch.from_numpy(c["mask"]).cuda(), symmetry="C3", wedge_box=nw)
        for i in range(0, 24, step):
            j = slice(i, i + step)
            kept = av.add(torch.from_numpy(c["parts"][j]).cuda(), c["rots"][j], c["halves"][j], shifts=c["shifts"][j],
                          weights=c["weights"][j], wedges=torch.from_numpy(c["wedges"]).cuda(), wedge_index=c["widx"][j])
            assert kept.all()
        sums.append([[t.cpu().numpy() for t in av.result(h)[:2]] for h in (1, 2)])
        av.close()
    for a, b in zip(*sums):
        assert np.abs(a[0] - b[0]).max() <= 4 * 12 * 2.0 ** -24 * np.abs(a[0]).max()
        assert np.array_equal(a[1], b[1])
