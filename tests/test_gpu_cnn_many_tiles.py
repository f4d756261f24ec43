"""Weight gradient over more tiles than the GPU takes at once: a block walks every 296th tile and
adds its sums to memory every four tiles.  The error is made zero outside chosen tiles, so that
the gradient is theirs alone and any one of the walk's stages shows: tiles of the first round,
of the second, of the fifth (after a flush), the last ones.  Against the float64 reference with
BF16-rounded weights and inputs: activations and output gradients are rounded to BF16 (2^-9
relative) at each of the four layers, 3e-2 as in the other gradient tests."""
import numpy as np
import pytest

from oracle import cnn_ref

pytestmark = pytest.mark.gpu

BLOCKS = 296                       # two per multiprocessor
SHAPE = (17, 1, 3005)              # tiles of 16 x 8 x 4: 2 x 1 x 752 = 1504, ragged in x, y and z


def _tile_of_cell():
    nx, ny, nz = SHAPE
    z, y, x = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    tx, ty = -(-nx // 16), -(-ny // 8)
    return x // 16 + tx * (y // 8 + ty * (z // 4))


def _reference(layers, x, dz_out):
    """Gradients of the float64 network for a given output gradient."""
    Ws = [(cnn_ref.bf16(W), np.asarray(b, np.float64)) for W, b in layers]
    a, zs = [cnn_ref.bf16(x)], []
    for l in range(4):
        zs.append(cnn_ref.conv(a[-1], *Ws[l]))
        if l < 3:
            a.append(cnn_ref.gelu(zs[-1]))
    ders = [cnn_ref.gelu_d(z) for z in zs[:3]]

    def backward(dz_channel):
        dz = np.zeros_like(zs[-1])
        dz[..., 0] = dz_channel
        grads = [None] * 4
        for l in range(3, -1, -1):
            grads[l] = cnn_ref.wgrad(dz, a[l])
            if l > 0:
                dz = cnn_ref.conv_t(dz, Ws[l][0]) * ders[l - 1]
        return grads
    return [backward(d) for d in dz_out]


def test_gradient_walks_all_tiles():
    from msg123_b200.learned import Cnn, unpack
    nx, ny, nz = SHAPE
    n = nx * ny * nz
    rng = np.random.default_rng(1)
    x = np.zeros((nz, ny, nx, 16), np.float32)
    x[..., :7] = rng.standard_normal((nz, ny, nx, 7))
    layers = []
    for l in range(4):
        W, b = np.zeros((27, 16, 16), np.float32), np.zeros(16, np.float32)
        co, ci = (1 if l == 3 else 16), (7 if l == 0 else 16)
        W[:, :co, :ci] = 0.15 * rng.standard_normal((27, co, ci))
        b[:co] = 0.05 * rng.standard_normal(co)
        layers.append((W, b))
    cnn = Cnn(seed=1)
    cnn.set_weights(np.concatenate([np.concatenate([W.reshape(-1), b]) for W, b in layers]).astype(np.float32))
    cnn.add_sample(SHAPE, x.reshape(-1, 16), np.zeros(n, np.float32))
    out = cnn.loss_grad(0, want_out=True, n=n)[2].reshape(nz, ny, nx)
    tile = _tile_of_cell()
    ntiles = tile.max() + 1
    assert ntiles == 1504 and ntiles % BLOCKS
    err = rng.standard_normal(out.shape).astype(np.float32)
    chosen = [tile < BLOCKS, (tile >= BLOCKS) & (tile < 2 * BLOCKS), (tile >= 3 * BLOCKS) & (tile < 4 * BLOCKS),
              tile >= 4 * BLOCKS, tile >= ntiles - 2, tile >= 0]
    errs = [np.where(m, err, np.float32(0)).astype(np.float32) for m in chosen]
    want = _reference(layers, x, [2.0 * e.astype(np.float64) / n for e in errs])
    for k, (e, ref) in enumerate(zip(errs, want)):
        cnn.add_sample(SHAPE, x.reshape(-1, 16), (out - e).reshape(-1))
        _, grad, again = cnn.loss_grad(k + 1, want_out=True, n=n)
        assert np.array_equal(again.reshape(out.shape), out)
        assert np.array_equal(cnn.loss_grad(k + 1)[1], grad)
        for l, ((gw, gb), (rw, rb)) in enumerate(zip(unpack(grad), ref)):
            co, ci = (1 if l == 3 else 16), (7 if l == 0 else 16)
            for a, r in ((gw[:, :co, :ci], rw[:, :co, :ci]), (gb[:co], rb[:co])):
                assert np.linalg.norm(a - r) <= 3e-2 * np.linalg.norm(r) + 1e-12, (k, l)
    cnn.close()
