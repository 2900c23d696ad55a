"""The learned tile proposal's CUDA kernels through the C ABI against the FP64 oracle (oracle/proposal.py): crop
features bit for bit, the training step's loss and gradients (FP32 on the device against FP64, tolerance stated per
check), Adam's update, the fused tensor-core prediction per tile, and the per-tile c-value sums that label the tiles."""

import numpy as np
import pytest

import es_b200
import es_synth
import oracle
import proposal
from gpu_util import from_dev, to_dev, zeros_dev

pytestmark = pytest.mark.gpu


def words_of(cuda, module, y, depth=10):
    """A CAMBI instance run on picture y; returns (instance, scale-0 words as numpy)."""
    h, w = y.shape
    c = es_b200.Cambi(module, w, h, depth)
    t = to_dev(cuda, y)
    c.launch(t.data_ptr(), w, cuda.cuda.current_stream().cuda_stream)
    c.finish()
    img, mask = c.read_scale(0)
    return c, (img.astype(np.uint16) | (mask.astype(np.uint16) << 15)), t


def needs_cvalue(words, p):
    code = (words & 0x7FFF).astype(np.int64) - p.band_base
    ok = ((words & 0x8000) != 0) & (code >= 0) & (code < p.band_size)
    value = code + p.band_base + 4
    need = np.zeros(words.shape, bool)
    for d in range(4):
        need |= (value <= p.tvi[d]) & (value + d + 1 > p.vlt)
    return ok & need


def random_params(seed):
    rng = np.random.default_rng(seed)
    params = proposal.init_params(seed)
    return [(w, (0.05 * rng.normal(size=b.shape)).astype(np.float32)) for w, b in params]


def test_features_match_the_oracle(cuda, module):
    step = es_synth.c2_step(0, w=300, h=200, n_encodes=1)
    c, words, keep = words_of(cuda, module, step.encodes[0].y)
    wd = to_dev(cuda, words)
    xy = np.array([[0, 0], [-16, -16], [100, 40], [290, 190], [-8, 120]], np.int32)
    n, fw, fh = len(xy), 24, 24
    out = zeros_dev(cuda, (n, 2, fh, fw), np.float32)
    es_b200.proposal_features(wd.data_ptr(), 300, 200, to_dev(cuda, xy).data_ptr(), n, fw, fh, out.data_ptr())
    got = from_dev(out, np.float32)
    for i, (x0, y0) in enumerate(xy):
        want = proposal.features_fast(words, int(x0), int(y0), fw, fh).astype(np.float32)
        assert np.array_equal(got[i], want), i
    c.close()


def test_training_step_gradients_match_the_oracle(cuda, module):
    rng = np.random.default_rng(11)
    n, size = 3, 8 + 2 * 16
    x = rng.normal(0, 1, (n, 2, size, size)).astype(np.float32)
    labels = rng.normal(0.5, 0.5, (n, 2, 2)).astype(np.float32)
    params = random_params(5)
    net = es_b200.ProposalNet(proposal.flatten(params))
    xd, ld = to_dev(cuda, x), to_dev(cuda, labels)
    loss, grads = net.train_step(xd.data_ptr(), ld.data_ptr(), n, size, size, 0.0, want_grads=True)
    want_loss, want = proposal.loss_and_grads(x.astype(np.float64), labels.astype(np.float64), params)
    assert abs(loss - want_loss) <= 1e-5 * abs(want_loss)
    want_flat = proposal.flatten([(gw, gb) for gw, gb in want]).astype(np.float64)
    # FP32 sums of ~4000 products against FP64: within 1e-3 of the largest gradient of the same layer
    at = 0
    for (gw, gb) in want:
        for g in (gw, gb):
            seg = slice(at, at + g.size)
            scale = np.abs(want_flat[seg]).max()
            assert np.abs(grads[seg] - want_flat[seg]).max() <= 1e-3 * scale + 1e-9
            at += g.size
    # the Adam step of the device from those gradients equals the oracle's Adam on the same gradients
    loss2, _ = net.train_step(xd.data_ptr(), ld.data_ptr(), n, size, size, 1e-3)
    got = net.params()
    opt = proposal.Adam(params, lr=1e-3)
    new = opt.step(params, proposal.unflatten(grads.astype(np.float64)))
    want_p = proposal.flatten(new)
    assert np.allclose(got, want_p, rtol=0, atol=2e-7)
    net.close()


def test_training_lowers_the_loss_on_the_device(cuda, module):
    rng = np.random.default_rng(3)
    n, size = 8, 8 + 2 * 16
    x = rng.normal(0, 1, (n, 2, size, size)).astype(np.float32)
    labels = np.tanh(x[:, 0, 8:-8:16, 8:-8:16] + 0.5 * x[:, 1, 8:-8:16, 8:-8:16]).astype(np.float32)  # a learnable target
    net = es_b200.ProposalNet(seed=1)
    xd, ld = to_dev(cuda, x), to_dev(cuda, labels)
    first, _ = net.train_step(xd.data_ptr(), ld.data_ptr(), n, size, size, 3e-3)
    for _ in range(150):
        last, _ = net.train_step(xd.data_ptr(), ld.data_ptr(), n, size, size, 3e-3)
    assert last < 0.3 * first
    net.close()


def test_prediction_matches_the_oracle(cuda, module):
    w, h = 330, 200
    step = es_synth.c2_step(1, w=w, h=h, n_encodes=3)
    c, words, keep = words_of(cuda, module, step.encodes[2].y)
    p = oracle.cambi_params(w, h)
    params = random_params(7)
    net = es_b200.ProposalNet(proposal.flatten(params))
    wd = to_dev(cuda, words)
    tx, ty = (w + 63) // 64, (h + 63) // 64
    pred = zeros_dev(cuda, (ty, tx), np.float32)
    net.predict(wd.data_ptr(), w, h, pred.data_ptr())
    got = from_dev(pred, np.float32)
    need = needs_cvalue(words, p)
    errs = []
    for j in range(ty):
        for i in range(tx):
            if not need[64 * j:64 * j + 64, 64 * i:64 * i + 64].any():
                assert got[j, i] == -np.inf, (i, j)
                continue
            f = proposal.features_fast(words, 64 * i - 16, 64 * j - 16, 24, 24)[None]
            z = proposal.forward(f.astype(np.float32).astype(np.float64), params, round_acts=True)[-1]
            want = z[0, 0].mean()
            errs.append(abs(got[j, i] - want))
    assert errs, "no tile needs c-values"
    # bfloat16 activations: an FP32 sum on either side of a rounding tie can move an activation by one bfloat16 step
    assert max(errs) <= 2e-2 and np.median(errs) <= 1e-3, (max(errs), np.median(errs))
    net.close()
    c.close()


def test_tile_masses_sum_the_cvalues_of_each_tile(cuda, module):
    w, h = 260, 150
    step = es_synth.c2_step(2, w=w, h=h, n_encodes=3)
    y = step.encodes[2].y
    n_tiles = es_b200.cambi_tile_count(w, h)
    c = es_b200.Cambi(module, w, h, 10)
    mass = zeros_dev(cuda, (n_tiles,), np.uint64)
    sizes = []
    ww, hh = w, h
    for _ in range(5):
        sizes.append((ww, hh))
        ww, hh = (ww + 1) >> 1, (hh + 1) >> 1
    planes = [zeros_dev(cuda, (sh, sw), np.float32) for sw, sh in sizes]
    c.set_tile_mass(mass.data_ptr())
    c.set_cvalue_planes([t.data_ptr() for t in planes])
    t = to_dev(cuda, y)
    c.launch(t.data_ptr(), w, cuda.cuda.current_stream().cuda_stream)
    c.finish()
    got = from_dev(mass, np.uint64)
    _, sums, _ = c.scale_stats()
    at = 0
    for s, (sw, sh) in enumerate(sizes):
        cv = from_dev(planes[s], np.float32).astype(np.float64)
        nx, ny = (sw + 63) // 64, (sh + 63) // 64
        for j in range(ny):
            for i in range(nx):
                blk = cv[64 * j:64 * j + 64, 64 * i:64 * i + 64]
                assert got[at + j * nx + i] == int(round((blk[blk > 0] * 16777216.0).sum())), (s, i, j)
        assert int(got[at:at + nx * ny].sum()) == sums[s]
        at += nx * ny
    assert at == n_tiles and got.sum() > 0
    c.close()


@pytest.mark.parametrize("n,th,tw", [(1, 1, 1), (3, 1, 2), (2, 3, 1), (5, 2, 4)])
def test_gradients_of_crops_around_the_weight_kernels_tiles(cuda, module, n, th, tw):
    """The weight gradients come from tiles of 8 x 36 output pixels: crops smaller than one, a little larger, and not
    square. Tolerance as above: FP32 sums of some thousand products against FP64."""
    rng = np.random.default_rng(n + 10 * th + 100 * tw)
    h, w = 8 + 16 * th, 8 + 16 * tw
    x = rng.normal(0, 1, (n, 2, h, w)).astype(np.float32)
    labels = rng.normal(0.5, 0.5, (n, th, tw)).astype(np.float32)
    params = random_params(6)
    net = es_b200.ProposalNet(proposal.flatten(params))
    xd, ld = to_dev(cuda, x), to_dev(cuda, labels)
    loss, grads = net.train_step(xd.data_ptr(), ld.data_ptr(), n, h, w, 0.0, want_grads=True)
    net.close()
    want_loss, want = proposal.loss_and_grads(x.astype(np.float64), labels.astype(np.float64), params)
    assert abs(loss - want_loss) <= 1e-5 * abs(want_loss)
    at = 0
    for gw, gb in want:
        for g in (gw, gb):
            got = grads[at:at + g.size].reshape(g.shape)
            assert np.abs(got - g).max() <= 1e-3 * np.abs(g).max() + 1e-9
            at += g.size


@pytest.mark.parametrize("n,th,tw", [(1, 1, 1), (2, 2, 2), (1, 4, 4)])
def test_an_infinite_input_reaches_only_the_taps_that_read_it(cuda, module, n, th, tw):
    """The last pixel of a crop's first channel is read by one tap of the first layer. Infinite there (and masked by the
    ReLU behind it, so that everything else stays finite), it makes that tap's weight gradients NaN (0 x inf) and leaves
    every other gradient as a finite value in its place leaves it, whatever the weight kernel's tiles reach past a crop."""
    rng = np.random.default_rng(n + th + tw)
    h, w = 8 + 16 * th, 8 + 16 * tw
    params = random_params(8)
    params[0][0][:, 0, 2, 2] = 0.5
    xd = rng.normal(0, 1, (n, 2, h, w)).astype(np.float32)
    ld = to_dev(cuda, rng.normal(0.5, 0.5, (n, th, tw)).astype(np.float32))
    grads = []
    for corner in (-1e4, -np.inf):
        xd[:, 0, h - 1, w - 1] = corner
        net = es_b200.ProposalNet(proposal.flatten(params))
        x = to_dev(cuda, xd)
        _, g = net.train_step(x.data_ptr(), ld.data_ptr(), n, h, w, 0.0, want_grads=True)
        grads.append(np.array(g))
        net.close()
    hit = np.zeros(grads[0].shape, bool)
    hit[:16 * 2 * 9].reshape(16, 2, 3, 3)[:, 0, 2, 2] = True
    assert np.isfinite(grads[0]).all() and np.isnan(grads[1][hit]).all()
    assert np.array_equal(grads[1][~hit], grads[0][~hit])


@pytest.mark.parametrize("n,th,tw", [(16, 4, 4), (40, 2, 5), (32, 4, 4)])
def test_gradients_of_batches_around_two_pixels_a_thread(cuda, module, n, th, tw):
    """The convolutions' threads make two pixels each in large batches: batches where the forward layers do and the backward
    ones do not, and where both do. Tolerances as above."""
    rng = np.random.default_rng(n)
    h, w = 8 + 16 * th, 8 + 16 * tw
    x = rng.normal(0, 1, (n, 2, h, w)).astype(np.float32)
    labels = rng.normal(0.5, 0.5, (n, th, tw)).astype(np.float32)
    params = random_params(7)
    net = es_b200.ProposalNet(proposal.flatten(params))
    xd, ld = to_dev(cuda, x), to_dev(cuda, labels)
    loss, grads = net.train_step(xd.data_ptr(), ld.data_ptr(), n, h, w, 0.0, want_grads=True)
    net.close()
    want_loss, want = proposal.loss_and_grads(x.astype(np.float64), labels.astype(np.float64), params)
    assert abs(loss - want_loss) <= 1e-5 * abs(want_loss)
    at = 0
    for gw, gb in want:
        for g in (gw, gb):
            got = grads[at:at + g.size].reshape(g.shape)
            assert np.abs(got - g).max() <= 1e-3 * np.abs(g).max() + 1e-9
            at += g.size


@pytest.mark.parametrize("n,th,tw", [(1, 2, 2), (4, 2, 2), (2, 4, 4)])
def test_gradients_of_a_flat_crop_round_like_short_chains(cuda, module, n, th, tw):
    """On a flat crop every product of a tap is the same number and additions in one long chain all round the same way. The
    network passes its first input through (middle taps 1), input, labels and number of tiles are such that everything up to
    the products is exact in FP32, so a gradient's only errors are its additions': 36 products in a row at most, then
    FP64 and three roundings to FP32 on the way, 40 half-steps of 2^-23 in all."""
    h, w = 8 + 16 * th, 8 + 16 * tw
    c, d = 507 / 512, 15347 / 16384
    params = [(np.zeros_like(a), np.zeros_like(b)) for a, b in random_params(1)]
    for weights, _ in params:
        weights[0, 0, 1, 1] = 1.0
    x = np.zeros((n, 2, h, w), np.float32)
    x[:, 0] = c
    labels = np.full((n, th, tw), c - d, np.float32)
    net = es_b200.ProposalNet(proposal.flatten(params))
    xd, ld = to_dev(cuda, x), to_dev(cuda, labels)
    _, grads = net.train_step(xd.data_ptr(), ld.data_ptr(), n, h, w, 0.0, want_grads=True)
    net.close()
    _, want = proposal.loss_and_grads(x.astype(np.float64), labels.astype(np.float64), params)
    want = np.concatenate([g.ravel() for pair in want for g in pair])
    assert want.min() >= 0 and (want > 0).sum() >= 40
    assert (np.abs(np.array(grads, np.float64) - want) <= 40 * 2.0 ** -24 * want).all()
