"""Learned-proposal form, training side, on the GPU: exact targets from the plain method, the
hand-written forward/backward kernels against a float64 CPU restatement, and training."""
import ctypes

import numpy as np
import pytest
import torch

import learned_ref
import pseudoctimaging_b200 as pct

pytestmark = pytest.mark.gpu
NP = pct.lib.pct_model_num_params()


def make_subjects(specs):
    subs, keep, host = [], [], []
    for nx, ny, nz, num, seed in specs:
        s = pct.synth_subject(nx, ny, nz, num, n_blobs=10, seed=seed)
        d = [torch.from_numpy(s.img).cuda(), torch.from_numpy(s.atlas_mri).cuda()]
        keep.append(d)
        host.append(s)
        subs.append(pct.TrainSubject(img=d[0].data_ptr(), atlas=d[1].data_ptr(), nx=nx, ny=ny,
                                     nz=nz, num_atlas=num))
    return subs, keep, host


def random_samples(host, n, seed):
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(n):
        s = int(rng.integers(len(host)))
        nz, nx, ny = host[s].img.shape
        a = int(rng.integers(host[s].atlas_mri.shape[0]))
        z, x, y = (int(rng.integers(6, d - 6)) for d in (nz, nx, ny))
        out.append((s, a, (z * nx + x) * ny + y))
    return np.array(out, np.int32)


class TrainSet:
    def __init__(self, subs, samples):
        arr = (pct.TrainSubject * len(subs))(*subs)
        ts = ctypes.c_void_p()
        st = pct.lib.pct_train_set_create(0, arr, len(subs), samples.ctypes.data, len(samples),
                                          ctypes.byref(ts))
        assert st == 0, st
        self.ptr, self.n = ts, len(samples)

    def targets(self):
        t = np.empty((self.n, 33), np.float32)
        top = np.empty((self.n, 32), np.int16)
        assert pct.lib.pct_train_set_targets(self.ptr, t.ctypes.data, top.ctypes.data) == 0
        return t, top

    def close(self):
        pct.lib.pct_train_set_destroy(self.ptr)


class Model:
    def __init__(self, seed):
        m = ctypes.c_void_p()
        assert pct.lib.pct_model_create(0, seed, ctypes.byref(m)) == 0
        self.ptr = m

    def params(self, inference=False):
        p = np.empty(NP, np.float32)
        assert pct.lib.pct_model_get_params(self.ptr, p.ctypes.data, int(inference)) == 0
        return p

    def grads(self, ts, begin, count):
        g = np.empty(NP, np.float32)
        loss = ctypes.c_float()
        assert pct.lib.pct_model_gradients(self.ptr, ts.ptr, begin, count, g.ctypes.data,
                                           ctypes.byref(loss)) == 0
        return loss.value, g

    def train(self, ts, batch, steps, lr):
        loss = ctypes.c_float()
        assert pct.lib.pct_model_train(self.ptr, ts.ptr, batch, steps, lr, ctypes.byref(loss)) == 0
        return loss.value

    def close(self):
        pct.lib.pct_model_destroy(self.ptr)


@pytest.fixture(scope="module")
def data():
    subs, keep, host = make_subjects([(40, 44, 36, 3, 31), (38, 36, 34, 2, 32)])
    yield subs, keep, host


def test_targets_are_the_plain_methods_top32(data):
    subs, keep, host = data
    samples = random_samples(host, 64, 1)
    ts = TrainSet(subs, samples)
    t, top = ts.targets()
    ts.close()
    np.testing.assert_allclose(t.reshape(-1, 3, 11).sum(axis=2), 1.0, atol=1e-5)
    for i, (s, a, vox) in enumerate(samples[:24]):
        ssd = learned_ref.top32_float64(host[s].img, host[s].atlas_mri[a], int(vox))
        order = np.sort(ssd)
        kth, nxt = order[31], order[32]
        chosen = ssd[top[i].astype(int)]
        # every GPU choice is among the 32 smallest (FP32 vs FP64 may swap near-ties at the edge)
        assert chosen.max() <= kth + 1e-4 * max(1.0, kth) or np.isclose(kth, nxt, rtol=1e-5)
        assert len(set(top[i].tolist())) == 32


def test_gradients_match_float64_restatement(data):
    subs, keep, host = data
    samples = random_samples(host, 6, 2)
    ts = TrainSet(subs, samples)
    t, _ = ts.targets()
    m = Model(7)
    loss, g = m.grads(ts, 0, len(samples))
    w = m.params(inference=True)  # the BF16 weights the kernels use
    x = learned_ref.patches([h.img for h in host], [h.atlas_mri for h in host], samples, None)
    ref_loss, ref_g = learned_ref.loss_and_grads(w, x, t)
    m.close()
    ts.close()
    assert loss == pytest.approx(ref_loss, rel=1e-4)
    rel = np.linalg.norm(g - ref_g) / np.linalg.norm(ref_g)
    assert rel < 1e-4, rel
    # layer by layer
    o = 0
    for name, shape in learned_ref.SIZES:
        n = int(np.prod(shape))
        a, b = g[o:o + n], ref_g[o:o + n]
        if np.linalg.norm(b) > 1e-9:
            assert np.linalg.norm(a - b) / np.linalg.norm(b) < 1e-3, name
        o += n


def test_training_reduces_the_loss(data):
    subs, keep, host = data
    samples = random_samples(host, 1024, 3)
    ts = TrainSet(subs, samples)
    m = Model(11)
    l0, _ = m.grads(ts, 0, 1024)
    m.train(ts, 128, 40, 3e-3)
    l1, _ = m.grads(ts, 0, 1024)
    m.close()
    ts.close()
    assert l1 < 0.9 * l0, (l0, l1)


@pytest.mark.parametrize("begin,count", [(0, 1), (3, 2), (1, 4), (0, 148), (5, 149), (2, 446)])
def test_gradients_at_every_fill_of_a_pass(data, begin, count):
    """Sample counts that leave a CTA's pass part-empty, give some CTAs one sample more than others,
    or one sample each; float64 bound from the FP32 sums of the layer-wise check above."""
    subs, keep, host = data
    samples = random_samples(host, 450, 4)
    ts = TrainSet(subs, samples)
    t, _ = ts.targets()
    m = Model(9)
    loss, g = m.grads(ts, begin, count)
    w = m.params(inference=True)
    m.close()
    ts.close()
    pick = slice(begin, begin + count)
    x = learned_ref.patches([h.img for h in host], [h.atlas_mri for h in host], samples[pick], None)
    ref_loss, ref_g = learned_ref.loss_and_grads(w, x, t[pick])
    assert loss == pytest.approx(ref_loss, rel=1e-4)
    assert np.linalg.norm(g - ref_g) / np.linalg.norm(ref_g) < 1e-4
