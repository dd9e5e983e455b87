"""The tensor-core key switch and packing (128- and 256-row tiles, the digits'
sum in parts, the rows in passes) against the CUDA-core kernels, bit for bit:
integer sums modulo 2^32 and 2^64, so no tolerance."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from tfhe_b200 import client, client64, lstm, torus64        # noqa: E402
from tfhe_b200.engine import Keys                           # noqa: E402
from tfhe_b200.params import ParamSet                       # noqa: E402


def _draw(shape, dtype, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    info = torch.iinfo(dtype)
    x = torch.randint(info.min, info.max, shape, device="cuda", generator=g, dtype=dtype)
    x.view(-1)[:1] = info.min                                # q / 2 itself
    return x


# (n, n_big = N, levels, base): one part and several, K blocks that the digits
# do not fill (N l % 128), a single K block
@pytest.mark.parametrize("n,N,l,log2_beta", [(742, 2048, 5, 4), (630, 1024, 5, 3), (63, 128, 1, 7), (64, 256, 3, 2)])
def test_keyswitch_matches_cuda_cores(n, N, l, log2_beta):
    p = ParamSet("ks", N=N, n=n, log2_beta_bs=7, l_bs=1, collapse=1, log2_beta_ks=log2_beta, l_ks=l,
                 sigma_glwe=1.0, sigma_lwe=2.0 ** 15)
    rng = np.random.default_rng(n)
    words = lambda shape: rng.integers(0, 2 ** 32, size=shape, dtype=np.uint64).astype(np.uint32)
    G, M = n // p.collapse, 2 ** p.collapse
    keys = Keys.create(p, np.zeros((2, 2, G * M, 1, N), dtype=np.uint32), words((l, N, n)), words((l, N)))
    for i, batch in enumerate([1, 127, 128, 129, 256, 257, 1185, 20001 if N == 2048 else 3001]):
        a, b = _draw((batch, N), torch.int32, i), _draw((batch,), torch.int32, 100 + i)
        keys.set_tuning()
        got = keys.keyswitch(a, b)
        keys.set_tuning(ks_tensor_cores=0)
        want = keys.keyswitch(a, b)
        keys.set_tuning()
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1]), batch
        in_place = b.clone()
        again = keys.keyswitch(a, in_place, b_out=in_place)
        assert torch.equal(again[0], want[0]) and torch.equal(in_place, want[1]), batch


@pytest.mark.parametrize("n,N,l", [(70, 1024, 5), (33, 128, 1)])
def test_keyswitch64_matches_cuda_cores(n, N, l):
    p = client64.Params64("ks64", N=N, n=n, log2_beta_bs=13, l_bs=2, collapse=1, log2_beta_ks=4, l_ks=l,
                          sigma_glwe=2.0 ** 17, sigma_lwe=2.0 ** 40)
    keys = torus64.Keys64(client64.keygen(p, 3))
    for i, batch in enumerate([1, 128, 129, 1500]):
        a, b = _draw((batch, N), torch.int64, i), _draw((batch,), torch.int64, 100 + i)
        got = keys.keyswitch(a, b, tensor_cores=1)
        want = keys.keyswitch(a, b, tensor_cores=0)
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1]), batch


@pytest.mark.parametrize("N,l,log2_beta", [(1024, 4, 7), (128, 3, 4)])
def test_packing_matches_cuda_cores(N, l, log2_beta):
    rng = np.random.default_rng(N)
    ksp = rng.integers(0, 2 ** 32, size=(N, l, 2, N), dtype=np.uint64).astype(np.uint32)
    key = lstm.PackingKey(ksp, log2_beta, l)
    assert key.tensor_cores
    for S, T in [(1, 1), (3, 43), (2, N), (9, 128), (20, 100)]:
        a, b = _draw((S, T, N), torch.int32, S), _draw((S, T), torch.int32, 100 + S)
        assert torch.equal(key.pack(a, b, tensor_cores=1), key.pack(a, b, tensor_cores=0)), (S, T)
