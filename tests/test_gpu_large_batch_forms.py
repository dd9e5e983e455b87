"""The large-batch forms of the blind rotation (several ciphertexts per CTA
sharing each key word) against the one-ciphertext-per-CTA form, bit for bit:
the same operations on every value, so no tolerance."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from tfhe_b200 import client, client64                      # noqa: E402
from tfhe_b200.engine import Keys                           # noqa: E402
from tfhe_b200.params import ParamSet                       # noqa: E402


def _batches():
    """One round of four per SM less and more one, the remainders on either
    side of each choice of form, and several rounds."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return [sms + 1, 2 * sms, 2 * sms + 1, 3 * sms, 3 * sms + 1, 4 * sms - 1, 4 * sms, 4 * sms + 1, 9 * sms + 3]


def _compare(keys, p, word, n, batch, n_lut, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    info = torch.iinfo(word)
    draw = lambda shape: torch.randint(info.min, info.max, shape, device="cuda", generator=g, dtype=word)
    a, b = draw((batch, n)), draw((batch,))
    for count in (1, batch):
        lut = draw((count, 2, p.N))
        keys.set_tuning()
        got = keys.cuboot_merge(a, b, lut, n_lut)
        acc = keys.blind_rotate(a, b, lut, n_lut)
        keys.set_tuning(ciphertexts_per_cta=1)
        want = keys.cuboot_merge(a, b, lut, n_lut)
        acc1 = keys.blind_rotate(a, b, lut, n_lut)
        keys.set_tuning()
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1]), (batch, n_lut, count)
        assert torch.equal(acc, acc1), (batch, n_lut, count)


@pytest.mark.parametrize("collapse", [1, 2, 3, 4])
def test_n2048_l2_matches_one_per_cta(collapse):
    p = ParamSet("n12_N2048", N=2048, n=12, log2_beta_bs=15, l_bs=2, collapse=collapse, log2_beta_ks=4, l_ks=5,
                 sigma_glwe=1.0, sigma_lwe=2.0 ** 15)
    k = client.keygen(p, collapse)
    keys = Keys.create(p, k.bsk, k.ksk_a, k.ksk_b)
    for i, batch in enumerate(_batches()):
        _compare(keys, p, torch.int32, p.n, batch, (1, 4)[i % 2], 100 * collapse + i)


@pytest.mark.parametrize("collapse", [1, 3])
def test_n2048_l2_torus64_matches_one_per_cta(collapse):
    from tfhe_b200.torus64 import Keys64
    p = client64.Params64("n12_N2048_q64", N=2048, n=12, log2_beta_bs=13, l_bs=2, collapse=collapse, log2_beta_ks=4,
                          l_ks=5, sigma_glwe=2.0 ** 17, sigma_lwe=2.0 ** 40)
    keys = Keys64(client64.keygen(p, collapse))
    for i, batch in enumerate(_batches()):
        _compare(keys, p, torch.int64, p.n, batch, (1, 4)[i % 2], 100 * collapse + i)


@pytest.mark.parametrize("l_bs,log2_beta,collapse", [(3, 7, 3), (3, 8, 3), (3, 7, 2), (2, 8, 3), (2, 7, 2)])
def test_n1024_matches_one_per_cta(l_bs, log2_beta, collapse):
    """The matrix-instruction kernel: its products are the exact integers, so
    its words are the general kernel's although the sums run in another order."""
    p = ParamSet("n198_N1024", N=1024, n=198, log2_beta_bs=log2_beta, l_bs=l_bs, collapse=collapse, log2_beta_ks=3,
                 l_ks=5, sigma_glwe=2.0 ** 7, sigma_lwe=2.0 ** 17)
    k = client.keygen(p, 10 * l_bs + collapse)
    keys = Keys.create(p, k.bsk, k.ksk_a, k.ksk_b)
    # below a round: clusters of eight, four and two CTAs for four ciphertexts
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    small = [1, 3, 4, 5, sms // 4, sms // 2, sms // 2 + 1, sms - 20, sms]
    for i, batch in enumerate(small + _batches()):
        _compare(keys, p, torch.int32, p.n, batch, (1, 4)[i % 2], 100 * collapse + i)


@pytest.mark.parametrize("l_bs,log2_beta,collapse", [(3, 7, 3), (2, 8, 2), (3, 9, 3)])
def test_dropin_n1024_matches_native_words(l_bs, log2_beta, collapse):
    """multiply_seq_monomial from the reference's key spectra, over every form of
    the matrix-instruction kernels, against the native one-per-CTA kernel on the
    same key (base 2^9 keeps the general kernel on both sides)."""
    from tfhe_b200 import ops
    p = ParamSet("n66_N1024", N=1024, n=66 if collapse == 3 else 64, log2_beta_bs=log2_beta, l_bs=l_bs,
                 collapse=collapse, log2_beta_ks=3, l_ks=5, sigma_glwe=2.0 ** 7, sigma_lwe=2.0 ** 17)
    k = client.keygen(p, 5)
    keys = Keys.create(p, k.bsk, k.ksk_a, k.ksk_b)
    j = torch.arange(p.N, device="cuda", dtype=torch.float64)
    coeff = torch.from_numpy(client._centred(k.bsk)).cuda().to(torch.float64)          # (in, out, G M, l, N)
    four = torch.fft.fft(coeff * torch.exp(-1j * np.pi * j / p.N))[..., : p.N // 2].permute(1, 0, 3, 2, 4).contiguous()
    angle = (torch.arange(2 * p.N, device="cuda")[:, None] * (2 * torch.arange(p.N // 2, device="cuda") + 1)) % (2 * p.N)
    rot = torch.exp(-1j * np.pi * angle.to(torch.float64) / p.N)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    for batch in (1, 4, sms // 4, sms // 2 + 1, sms, 2 * sms, 4 * sms + 1):
        a = torch.randint(-2 ** 31, 2 ** 31 - 1, (batch, p.n), device="cuda", generator=g, dtype=torch.int32)
        for shared in (True, False):
            lut = torch.randint(-2 ** 31, 2 ** 31 - 1, (1 if shared else batch, 2, p.N), device="cuda", generator=g,
                                dtype=torch.int32)
            got = ops.multiply_seq_monomial(lut.to(torch.float64), a.to(torch.float64), four, 32, log2_beta, l_bs, p.N,
                                            collapse, rot, 2)
            keys.set_tuning(ciphertexts_per_cta=1)
            want = keys.blind_rotate(a, torch.zeros(batch, dtype=torch.int32, device="cuda"), lut, 2)
            keys.set_tuning()
            assert torch.equal((got.to(torch.int64) & 0xFFFFFFFF), (want.to(torch.int64) & 0xFFFFFFFF)), (batch, shared)


@pytest.mark.parametrize("torus", [32, 64])
@pytest.mark.parametrize("collapse", [2, 3])
def test_n2048_l2_small_batches_match_one_per_cta(torus, collapse):
    """Four ciphertexts per cluster of eight or four CTAs: whole and partly
    filled clusters, either side of each choice of form; 35 groups or more, so
    that the rotation indices' window moves."""
    word = torch.int32 if torus == 32 else torch.int64
    if torus == 32:
        p = ParamSet("n105_N2048", N=2048, n=35 * collapse, log2_beta_bs=15, l_bs=2, collapse=collapse, log2_beta_ks=4,
                     l_ks=5, sigma_glwe=1.0, sigma_lwe=2.0 ** 15)
        k = client.keygen(p, collapse)
        keys = Keys.create(p, k.bsk, k.ksk_a, k.ksk_b)
    else:
        from tfhe_b200.torus64 import Keys64
        p = client64.Params64("n105_N2048_q64", N=2048, n=35 * collapse, log2_beta_bs=13, l_bs=2, collapse=collapse,
                              log2_beta_ks=4, l_ks=5, sigma_glwe=2.0 ** 17, sigma_lwe=2.0 ** 40)
        keys = Keys64(client64.keygen(p, collapse))
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for i, batch in enumerate([1, 3, 4, 5, sms // 4, sms // 2 - 2, sms // 2 + 1, sms - 20, sms]):
        _compare(keys, p, word, p.n, batch, (1, 4)[i % 2], 10 * collapse + i)
