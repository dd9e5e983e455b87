"""The layer's linear and LUT products on both tori over their forms (sparse
and dense weights, one to four coefficients per thread, transform and direct
sums), against exact integer sums modulo 2^32 or 2^64."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from tfhe_b200 import lstm                                  # noqa: E402


def _negacyclic(w, x):
    """w (N) small integers, x (N) unsigned words -> w x mod X^N + 1."""
    N = len(x)
    out = np.zeros(N, dtype=x.dtype)
    for m in np.nonzero(w)[0]:
        rolled = np.concatenate([(0 - x[N - m:]).astype(x.dtype), x[: N - m]]) if m else x
        out += (np.array(int(w[m])).astype(np.int64).astype(x.dtype) * rolled).astype(x.dtype)
    return out


def _words(rng, shape, bits):
    u = rng.integers(0, 2 ** 64, size=shape, dtype=np.uint64)
    return u if bits == 64 else (u >> np.uint64(32)).astype(np.uint32)


def _dev(x, bits):
    return torch.from_numpy(np.ascontiguousarray(x).view(np.int64 if bits == 64 else np.int32)).cuda()


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("N,J,S,density", [(128, 1, 1, 1.0), (256, 5, 2, 0.0), (1024, 4, 3, 0.3), (2048, 9, 40, 0.05),
                                           (4096, 3, 1, 1.0)])
def test_linear_extract_exact(bits, N, J, S, density):
    rng = np.random.default_rng(N + J + S)
    w = rng.integers(-2 ** 31, 2 ** 31, size=(J, N)) * (rng.random((J, N)) < density)
    x = _words(rng, (S, 2, N), bits)
    bias = _words(rng, (J,), bits)
    a, b = lstm.linear_extract(torch.from_numpy(w.astype(np.int32)).cuda(), _dev(bias, bits), _dev(x, bits))
    a, b = a.cpu().numpy().view(x.dtype), b.cpu().numpy().view(x.dtype)
    for s in {0, S - 1}:
        for j in range(J):
            pa, pb = _negacyclic(w[j], x[s, 0]), _negacyclic(w[j], x[s, 1])
            want = np.concatenate([pa[:1], (0 - pa[:0:-1]).astype(x.dtype)])
            assert np.array_equal(a[s, j], want), (s, j)
            assert b[s, j] == (pb[:1] + bias[j: j + 1]).astype(x.dtype)[0], (s, j)


@pytest.mark.parametrize("N,G,most", [(128, 1, 128), (128, 1, 129), (1024, 4, 4), (1024, 4, 5), (2048, 3, 2),
                                      (2048, 16, 1), (4096, 2, 1)])
def test_lut_products_exact(N, G, most):
    """On either side of the bound G N max|LUT| = 2^14 of the transform."""
    rng = np.random.default_rng(N + G + most)
    K, S = 2, 2
    lut = rng.integers(-most, most + 1, size=(G, K, N))
    lut[0, :, 0] = -most
    x = _words(rng, (S, G, K, 2, N), 32)
    x[0, 0, 0] = 0x80000000                                   # the most negative word everywhere
    got = lstm.lut_mul_sum(torch.from_numpy(lut.astype(np.int32)).cuda(), _dev(x, 32)).cpu().numpy().view(np.uint32)
    for s in range(S):
        for k in range(K):
            for a in range(2):
                want = np.zeros(N, dtype=np.uint32)
                for g in range(G):
                    want += _negacyclic(lut[g, k], x[s, g, k, a])
                assert np.array_equal(got[s, k, a], want), (s, k, a)


@pytest.mark.parametrize("log2_beta,l", [(8, 5), (7, 6), (9, 4)])
def test_trace64_n2048_matches_general_kernel(monkeypatch, log2_beta, l):
    """The kernel of three limbs against the general one on the same keys, from
    one LWE to more than a round of CTAs; masks and bodies include zero, the
    most negative word, and multiples of a digit's half (ties)."""
    from tfhe_b200 import torus64
    N = 2048
    rng = np.random.default_rng(100 * l + log2_beta)
    keys = _words(rng, (11, l, 2, N), 64)
    keys[:, 0] = np.uint64(2 ** 64 - 2 ** 63 - 2 ** 42 - 2 ** 21)      # every limb at its largest
    here = torus64.GaloisKeys64(keys, log2_beta, l)
    monkeypatch.setenv("TFHE_B200_TRACE_TREE", "0")
    general = torus64.GaloisKeys64(keys, log2_beta, l)
    for R in (1, 3, 300):
        a, b = _words(rng, (R, N), 64), _words(rng, (R,), 64)
        a[0] = 0
        if R > 2:
            a[1] = 1 << 63
            a[2] <<= 63 - l * log2_beta + 11
            b[1] = 1 << 63
            a[-1] = a[-1, 0]                                           # digits that add up
        got = here.pack_lwe_to_rlwe(_dev(a, 64), _dev(b, 64))
        assert torch.equal(got, general.pack_lwe_to_rlwe(_dev(a, 64), _dev(b, 64))), R
