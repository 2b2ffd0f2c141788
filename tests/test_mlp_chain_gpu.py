"""gbsdf_mlp_chain against the same layers run one by one through gbsdf_dense: the same products,
accumulation order and roundings, so every half of every layer is equal bit for bit."""
import pytest
import torch

from neuralangelo_gb300 import fused
from neuralangelo_gb300.dense import EPI_IDENTITY, EPI_RELU, EPI_SOFTPLUS

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
SMS = 152
# per layer (width, input columns from memory, activation); a tile's edges, one tile per CTA and
# more, chains of two layers and more with one and two units of appended columns
FEATURE = [(256, 256, EPI_SOFTPLUS), (256, 48, EPI_RELU), (256, 0, EPI_RELU), (256, 0, EPI_RELU), (256, 0, EPI_RELU)]
SMALL = [(256, 256, EPI_SOFTPLUS), (128, 32, EPI_RELU), (128, 0, EPI_RELU)]
SKIP = [(256, 96, EPI_RELU)] + 3 * [(256, 0, EPI_RELU)] + [(256, 96, EPI_RELU)] + 3 * [(256, 0, EPI_RELU)] + [
    (128, 48, EPI_RELU)]
ODD = [(128, 16, EPI_IDENTITY), (256, 80, EPI_SOFTPLUS), (128, 128, EPI_RELU), (256, 0, EPI_IDENTITY)]
PAIR = [(256, 208, EPI_RELU), (128, 0, EPI_RELU)]


@pytest.mark.parametrize("shape,M", [(FEATURE, 1), (FEATURE, 127), (FEATURE, 128 * SMS + 65), (SMALL, 300),
                                     (SMALL, 128 * SMS * 2 + 1), (SKIP, 128 * SMS + 1), (SKIP, 500), (ODD, 129),
                                     (ODD, 128 * SMS * 3), (PAIR, 128 * SMS * 2 + 128)])
def test_chain_equals_layer_by_layer(shape, M):
    g = torch.Generator(DEV).manual_seed(M + len(shape))
    f16 = dict(device=DEV, dtype=torch.float16)

    def pair(cols, ld):
        x = torch.randn(M, ld, device=DEV, generator=g)
        hi = x.half()
        return hi[:, :cols], (x - hi.float()).half()[:, :cols]

    layers, want, got, err = [], [], [], torch.zeros(1, device=DEV, dtype=torch.int32)
    prev = None
    for i, (N, K_in, epi) in enumerate(shape):
        K = (shape[i - 1][0] if i else 0) + K_in
        W = (torch.randn(N, K, device=DEV, generator=g) * K ** -0.5).half()
        b = torch.randn(N, device=DEV, generator=g) * 0.1 if i % 3 != 2 else None
        inp = pair(K_in, K_in + 8 * (i % 2)) if K_in else None
        halves = [t for t in (prev, inp) if t is not None]
        X, Xl = (torch.cat([t[j] for t in halves], dim=1).contiguous() for j in (0, 1))
        Y, Yl = torch.empty(M, N, **f16), torch.empty(M, N, **f16)
        fused._dense(X, W, N, K, Y, bias=b, epi=epi, beta=100.0, X_lo=Xl, out_lo=Yl, err=err)
        want.append((Y, Yl))
        prev = (Y, Yl)
        buf = [torch.full((M, N + 8), -7.0, **f16) for _ in range(2)]
        o = buf[0] if i % 4 != 3 or i + 1 == len(shape) else None          # some layers stay on chip
        ol = buf[1] if i % 2 == 0 or o is None else None
        got.append((o, ol))
        layers.append((W, b, epi, (*inp, K_in) if inp else None, o, ol))
    fused._mlp_chain(layers, 100.0, err)
    torch.cuda.synchronize()
    assert err.item() == 0
    for (N, _, _), w, o in zip(shape, want, got):
        for a, b in zip(w, o):
            if b is not None:
                assert torch.equal(a, b[:, :N]) and bool((b[:, N:] == -7).all())


def test_chain_rejects_what_it_cannot_run():
    x = torch.zeros(8, 64, device=DEV, dtype=torch.float16)
    W = torch.zeros(64, 64, device=DEV, dtype=torch.float16)
    W2 = torch.zeros(128, 64, device=DEV, dtype=torch.float16)
    one = (W2, None, EPI_RELU, (x, x, 64), None, None)
    with pytest.raises(RuntimeError, match="width 64"):
        fused._mlp_chain([(W, None, EPI_RELU, (x, x, 64), None, None), one], 1.0, None)
    with pytest.raises(RuntimeError, match="layers"):
        fused._mlp_chain([one], 1.0, None)
