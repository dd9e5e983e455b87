"""Which form a call runs, and that every form a key set reaches gives the
one-ciphertext-per-CTA form's words, bit for bit."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from tfhe_b200.engine import Keys                           # noqa: E402
from tfhe_b200.params import ParamSet                       # noqa: E402


def _params(N, n, l_bs, log2_beta, collapse):
    return ParamSet(f"n{n}_N{N}_c{collapse}", N=N, n=n, log2_beta_bs=log2_beta, l_bs=l_bs, collapse=collapse,
                    log2_beta_ks=3, l_ks=2, sigma_glwe=1.0, sigma_lwe=1.0)


def _keys(p, seed=0):
    """Uniform words as keys: the forms compute on them as on real ones."""
    rng = np.random.default_rng(seed)
    words = lambda shape: rng.integers(0, 2 ** 32, size=shape, dtype=np.uint64).astype(np.uint32)
    return Keys.create(p, words((2, 2, p.G * p.M, p.l_bs, p.N)), words((p.l_ks, p.N, p.n)), words((p.l_ks, p.N)))


class Hog:
    """All of the GPU's memory but `leave` bytes, given back in steps."""

    def __init__(self, leave):
        torch.cuda.empty_cache()
        self.held = [torch.empty(torch.cuda.mem_get_info()[0] - leave, dtype=torch.uint8, device="cuda")]

    def leave(self, nbytes):
        del self.held[1:]
        torch.cuda.empty_cache()
        free = torch.cuda.mem_get_info()[0]
        if free > nbytes:
            self.held.append(torch.empty(free - nbytes, dtype=torch.uint8, device="cuda"))

    def close(self):
        self.held.clear()
        torch.cuda.empty_cache()


def _draw(shape, seed, dtype=torch.int32):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    info = torch.iinfo(dtype)
    return torch.randint(info.min, info.max, shape, device="cuda", generator=g, dtype=dtype)


def _same_as_one_per_cta(keys, batch, seed=0, tuning=(0, -1, -1)):
    p = keys.params
    a, b, lut = _draw((batch, p.n), seed), _draw((batch,), seed + 1), _draw((batch, 2, p.N), seed + 2)
    keys.set_tuning(*tuning)
    got = keys.cuboot_merge(a, b, lut)
    keys.set_tuning(ciphertexts_per_cta=1)
    want = keys.cuboot_merge(a, b, lut)
    keys.set_tuning()
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1]), batch


def test_key_sets_of_several_sizes_in_turn():
    """A cluster kernel's shared memory grows with the number of groups and
    patterns: a smaller key set in between leaves the larger one launchable."""
    large, small = _keys(_params(1024, 120, 3, 9, 2)), _keys(_params(1024, 24, 3, 9, 2))
    for keys in (large, small, large):
        for batch in (1, 60):                                # one ciphertext per cluster of eight, per pair
            _same_as_one_per_cta(keys, batch)


def test_keys_that_fit_without_the_second_layout():
    """The second layout of a key (N = 1024, base <= 2^8) takes only memory that
    the rest of the key set leaves: once a set fits, it fits with more memory
    too, and without the layout it gives the same words."""
    p = _params(1024, 120, 3, 7, 3).with_(l_ks=8)
    both = _keys(p)
    full = both.device_bytes()
    both.close()
    layout = p.bsk_bytes_fp64()
    hog = Hog(full + (64 << 20))
    fits, single = [], None
    try:
        for nbytes in range(layout, full + (32 << 20), 2 << 20):
            hog.leave(nbytes)
            try:
                keys = _keys(p)
            except Exception:
                assert not fits, (nbytes, fits)
                continue
            fits.append(nbytes)
            if keys.device_bytes() == full - layout:
                single = keys
            else:
                assert keys.device_bytes() == full
                keys.close()
                break
    finally:
        hog.close()
    assert single is not None
    for batch in (1, 30, 60, 140, 300):
        _same_as_one_per_cta(single, batch)


@pytest.mark.parametrize("N,n,l_bs,log2_beta,collapse", [(1024, 630, 3, 7, 3), (2048, 742, 2, 15, 2)])
@pytest.mark.parametrize("clusters", [1, 5])
def test_a_lost_message_ends_the_cluster(N, n, l_bs, log2_beta, collapse, clusters):
    """One message of group 1 never arrives.  The waits for it run out, then those
    for the CTAs that gave up, and the kernel ends: three limits of 1 ms and the
    stay of 1 ms behind them at most, 10 ms with the launch (to run out in every
    group would take hundreds).  Outputs stay, the status says so, the keys work."""
    import ctypes
    from tfhe_b200 import _lib
    lib = _lib.load()
    keys = _keys(_params(N, n, l_bs, log2_beta, collapse))
    batch = clusters * (4 if N == 1024 else 2)
    a, b, lut = _draw((batch, n), 1), _draw((batch,), 2), _draw((1, 2, N), 3)
    out_a = torch.full((batch, 1, N), 77, dtype=torch.int32, device="cuda")
    out_b = torch.full((batch, 1), 77, dtype=torch.int32, device="cuda")
    _same_as_one_per_cta(keys, batch)
    st = ctypes.c_int32()
    _lib.check(lib.tfhe_device_status(ctypes.byref(st), 1))
    t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    p = lambda x: ctypes.c_void_p(x.data_ptr())
    t0.record()
    _lib.check(lib.tfhe_probe_lost_message(keys.handle, p(a), p(b), p(lut), p(out_a), p(out_b), batch, 1_900_000,
                                           ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    t1.record()
    torch.cuda.synchronize()
    _lib.check(lib.tfhe_device_status(ctypes.byref(st), 1))
    assert st.value == 1
    assert t0.elapsed_time(t1) < 10.0
    assert bool((out_a == 77).all()) and bool((out_b == 77).all())
    _same_as_one_per_cta(keys, batch)


def _launched(keys, batch):
    """The number of kernels that a batch's blind rotation launches."""
    from tfhe_b200.engine import launch_count
    p = keys.params
    a, b, lut = _draw((batch, p.n), 1), _draw((batch,), 2), _draw((1, 2, p.N), 3)
    before = launch_count()
    keys.cuboot_merge(a, b, lut)
    return launch_count() - before


def _sizes(batch, sms):
    return batch if batch >= 0 else sms * -batch


# (degree, groups x collapse, levels, base, collapse), tuning, {batch (negative: x SMs): launches}
MMA = (1024, 24, 3, 7, 3)
FORMS = [
    (MMA, (0, -1, -1), {1: [(4, 8)], 37: [(4, 8)], 100: [(4, 4)], 200: [(4, 2)], -4: [(4, 1)], 593: [(4, 1), (4, 8)]}),
    (MMA, (0, -1, 0), {1: [(1, 8)], 24: [(1, 4)], 60: [(1, 2)], 148: [(1, 1)]}),
    (MMA, (2, -1, -1), {1: [(1, 1)], 200: [(2, 1)]}),
    ((1024, 24, 3, 9, 3), (0, -1, -1), {1: [(1, 8)], 24: [(1, 4)], 60: [(1, 2)], 148: [(1, 1)], 296: [(2, 1)]}),
    ((1024, 24, 2, 9, 2), (0, -1, -1), {1: [(1, 8)], 24: [(1, 4)], 60: [(1, 2)], 148: [(1, 1)]}),
    ((2048, 24, 2, 15, 2), (0, -1, -1), {1: [(1, 8)], 24: [(1, 4)], 56: [(2, 4)], 74: [(1, 2)], 148: [(1, 1)],
                                         -2: [(2, 1)], -4: [(4, 1)], 593: [(4, 1), (1, 8)]}),
]


@pytest.mark.parametrize("shape,tuning,batches", FORMS)
def test_launches_say_what_runs(shape, tuning, batches):
    """Batches for a GPU of 148 SMs; on another only the sums are checked."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    keys = _keys(_params(*shape))
    for batch, forms in batches.items():
        batch = _sizes(batch, sms)
        keys.set_tuning(*tuning)
        launches = keys.launches(batch)
        assert sum(x[0] for x in launches) == batch
        assert len(launches) == _launched(keys, batch)
        if sms == 148:
            assert [x[1:] for x in launches] == forms, (batch, launches)
        _same_as_one_per_cta(keys, batch, tuning=tuning)
    assert keys.launches(0) == []
    with pytest.raises(ValueError):
        keys.launches(-1)


def test_launches_say_what_runs64():
    from tfhe_b200 import client64
    from tfhe_b200.torus64 import Keys64
    p = client64.Params64("n24", N=2048, n=24, log2_beta_bs=13, l_bs=2, collapse=3, log2_beta_ks=4, l_ks=5,
                          sigma_glwe=2.0 ** 17, sigma_lwe=2.0 ** 40)
    keys = Keys64(client64.keygen(p, 3))
    for batch, forms in {1: [(1, 8)], 24: [(1, 4)], 56: [(2, 4)], 74: [(1, 2)], 148: [(1, 1)], 296: [(2, 1)],
                         592: [(4, 1)]}.items():
        launches = keys.launches(batch)
        a, b, lut = (_draw(s, 1, torch.int64) for s in ((batch, p.n), (batch,), (1, 2, p.N)))
        from tfhe_b200.engine import launch_count
        before = launch_count()
        keys.cuboot_merge(a, b, lut)
        assert len(launches) == launch_count() - before and sum(x[0] for x in launches) == batch
        if torch.cuda.get_device_properties(0).multi_processor_count == 148:
            assert [x[1:] for x in launches] == forms, (batch, launches)


@pytest.mark.parametrize("l_bs,collapse", [(3, 3), (3, 2), (2, 3), (2, 2)])
def test_n1024_general_kernels_between_the_clusters(l_bs, collapse):
    """The batches that the general kernels run sooner than the next wider
    clusters of four ciphertexts, alone and behind whole rounds, and the batches
    on either side of them."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    if sms != 148:
        pytest.skip("batches for a GPU of 148 SMs")
    keys = _keys(_params(1024, 24, l_bs, 7, collapse))
    for batch, forms in {40: [(4, 8)], 74: [(1, 2)], 75: [(4, 4)], 100: [(4, 4)], 148: [(1, 1)],
                         149: [(4, 2)], 592 + 74: [(4, 1), (1, 2)], 592 + 148: [(4, 1), (1, 1)]}.items():
        assert [x[1:] for x in keys.launches(batch)] == forms, (batch, keys.launches(batch))
        _same_as_one_per_cta(keys, batch)


@pytest.mark.parametrize("collapse", [2, 3, 4])
def test_n2048_two_per_cta_up_to_three_per_sm(collapse):
    """Few ciphertexts above two per SM do not pay for a round of four per CTA."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    keys = _keys(_params(2048, 24, 2, 15, collapse))
    for batch, first in {2 * sms + 1: (2 * sms, 2, 1), 3 * sms: (2 * sms, 2, 1), 3 * sms + 1: (3 * sms + 1, 4, 1),
                         6 * sms + 1: (4 * sms, 4, 1)}.items():
        launches = keys.launches(batch)
        assert launches[0] == first, (batch, launches)
        _same_as_one_per_cta(keys, batch)


@pytest.mark.parametrize("l_bs,log2_beta", [(1, 20), (2, 15), (3, 9)])
def test_fourier_key_is_the_coefficient_key(l_bs, log2_beta):
    """A key given as spectra lies in the order of the same key given as
    coefficients, at N = 2048 whatever the levels: the same accumulators."""
    from tfhe_b200 import client
    p = _params(2048, 8, l_bs, log2_beta, 2)
    rng = np.random.default_rng(l_bs)
    words = lambda shape: rng.integers(0, 2 ** 32, size=shape, dtype=np.uint64).astype(np.uint32)
    bsk, ka, kb = words((2, 2, p.G * p.M, l_bs, p.N)), words((p.l_ks, p.N, p.n)), words((p.l_ks, p.N))
    # small key words: both ways round to the same integers
    bsk = (bsk.view(np.int32) >> 16).view(np.uint32)
    j = np.arange(p.N)
    four = np.fft.fft(client._centred(bsk).astype(np.float64) * np.exp(-1j * np.pi * j / p.N))[..., : p.N // 2]
    ordered = np.ascontiguousarray(four.transpose(1, 0, 3, 2, 4))                   # (out, in, l, G M, N/2)
    one, two = Keys.create(p, bsk, ka, kb), Keys.create_fourier(p, ordered, ka, kb)
    for batch in (1, 30, 64, 148, 300, 600):
        a, b, lut = _draw((batch, p.n), 1), _draw((batch,), 2), _draw((1, 2, p.N), 3)
        x, y = one.blind_rotate(a, b, lut), two.blind_rotate(a, b, lut)
        assert torch.equal(x, y), batch


@pytest.mark.parametrize("n,N,l,log2_beta", [(63, 128, 1, 7), (63, 128, 3, 4), (100, 256, 1, 7), (200, 128, 4, 4)])
def test_short_key_switch_makes_its_digits_in_the_kernel(n, N, l, log2_beta):
    """One launch where one column tile (or few rows) uses the digits of a short
    sum, else the digit matrix and the sum; the CUDA cores' words either way."""
    from tfhe_b200.engine import launch_count
    p = ParamSet("ks", N=N, n=n, log2_beta_bs=7, l_bs=1, collapse=1, log2_beta_ks=log2_beta, l_ks=l, sigma_glwe=1.0,
                 sigma_lwe=1.0)
    keys = _keys(p)
    for batch in (1, 32, 33, 128, 129, 1000):
        a, b = _draw((batch, N), batch), _draw((batch,), 7)
        a.view(-1)[:1] = -2 ** 31
        before = launch_count()
        got = keys.keyswitch(a, b)
        short = N * l < 512 and (4 * (n + 1) <= 256 or batch <= 32)
        assert launch_count() - before == (1 if short else 2), batch
        keys.set_tuning(ks_tensor_cores=0)
        want = keys.keyswitch(a, b)
        keys.set_tuning()
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1]), batch


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("N", [128, 256, 512, 1024])
def test_linear_of_many_outputs_is_that_of_few(N, bits):
    """As many coefficients per thread as the degree has against one: exact sums,
    so the same words."""
    from tfhe_b200 import lstm
    dtype = torch.int32 if bits == 32 else torch.int64
    J, S = 1201, 2
    w, bias, x = _draw((J, N), 1), _draw((J,), 2, dtype), _draw((S, 2, N), 3, dtype)
    w[::3] = 0
    a, b = lstm.linear_extract(w, bias, x)
    for j in range(0, J, 100):
        pa, pb = lstm.linear_extract(w[j: j + 8].contiguous(), bias[j: j + 8].contiguous(), x)
        assert torch.equal(a[:, j: j + 8], pa) and torch.equal(b[:, j: j + 8], pb), j


FIRST_IN_CAPTURE = """
import sys, numpy as np, torch
sys.path[:0] = {paths!r}
from tfhe_b200 import lstm
N, G, K, S = {N}, 2, 3, 2
rng = np.random.default_rng(0)
lut = torch.from_numpy(rng.integers(-1, 2, size=(G, K, N)).astype(np.int32)).cuda()
x = torch.from_numpy(rng.integers(-2 ** 31, 2 ** 31, size=(S, G, K, 2, N)).astype(np.int32)).cuda()
out = torch.zeros((S, K, 2, N), dtype=torch.int32, device="cuda")
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    lstm.lut_mul_sum(lut, x, out=out)
graph.replay()
torch.cuda.synchronize()
first = out.clone()
assert torch.equal(lstm.lut_mul_sum(lut, x), first) and bool(first.any())
graph.replay()
torch.cuda.synchronize()
assert torch.equal(out, first)
print("equal")
"""


@pytest.mark.parametrize("N", [256, 2048])
def test_lut_products_first_called_in_a_capture(N):
    """Without keys of its degree in the process, the first call may be one being
    captured: direct sums there, the transform's words after it."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    code = FIRST_IN_CAPTURE.format(N=N, paths=[os.path.join(root, "blind-spiking-lstm_b200")])
    run = subprocess.run([sys.executable, "-c", code], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True,
                         timeout=300)
    assert run.returncode == 0 and run.stdout.strip().endswith("equal"), run.stdout


def _instantiated_twice(graph):
    """Two executables of one captured graph, each as a call that launches it and
    waits; the second instantiation is refused for a graph with memory nodes."""
    import ctypes
    rt = ctypes.CDLL("libcudart.so.12")
    execs = [ctypes.c_void_p(), ctypes.c_void_p()]
    for ex in execs:
        assert rt.cudaGraphInstantiate(ctypes.byref(ex), ctypes.c_void_p(graph.raw_cuda_graph()), ctypes.c_ulonglong(0)) == 0

    def launch(ex):
        assert rt.cudaGraphLaunch(ex, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
        torch.cuda.synchronize()

    for ex in execs:
        yield lambda: launch(ex)
    for ex in execs:
        assert rt.cudaGraphExecDestroy(ex) == 0


def test_a_captured_key_switch_adds_no_memory_nodes():
    """A graph with memory nodes is instantiated once only; that of a key switch
    twice, and both give the uncaptured call's words."""
    keys = _keys(_params(1024, 120, 1, 9, 2))
    a, b = _draw((200, 1024), 1), _draw((200,), 2)
    want = keys.keyswitch(a, b)
    out_a, out_b = torch.empty_like(want[0]), torch.empty_like(want[1])
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        keys.keyswitch(a, b, out_a, out_b)
    for launch in _instantiated_twice(graph):
        out_a.zero_()
        out_b.zero_()
        launch()
        assert torch.equal(out_a, want[0]) and torch.equal(out_b, want[1])


def _dropin(l_bs, log2_beta, collapse, n=24):
    """The drop-in's arguments (BSK, rot) for a uniform key of small words, as the
    reference holds them, at N = 1024."""
    N, G = 1024, n // collapse
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    coeff = torch.randint(-2 ** 15, 2 ** 15, (2, 2, G << collapse, l_bs, N), device="cuda", generator=g).to(torch.float64)
    j = torch.arange(N, device="cuda", dtype=torch.float64)
    four = torch.fft.fft(coeff * torch.exp(-1j * np.pi * j / N))[..., : N // 2].permute(1, 0, 3, 2, 4).contiguous()
    angle = (torch.arange(2 * N, device="cuda")[:, None] * (2 * torch.arange(N // 2, device="cuda") + 1)) % (2 * N)
    return four, torch.exp(-1j * np.pi * angle.to(torch.float64) / N)


@pytest.mark.parametrize("l_bs,collapse", [(3, 3), (3, 2), (2, 3), (2, 2)])
def test_a_captured_dropin_adds_no_memory_nodes(l_bs, collapse):
    """The drop-in reads its key in place in a capture and lays it out anew
    elsewhere: the same values, and a graph that is instantiated twice."""
    from tfhe_b200 import ops
    four, rot = _dropin(l_bs, 7, collapse)
    for batch in (1, 5, 150):
        a, lut = _draw((batch, 24), 1).to(torch.float64), _draw((batch, 2, 1024), 2).to(torch.float64)
        call = lambda: ops.multiply_seq_monomial(lut, a, four, 32, 7, l_bs, 1024, collapse, rot, 1)
        want = call()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph(keep_graph=True)
        with torch.cuda.graph(graph):
            out = call()
        for launch in _instantiated_twice(graph):
            out.zero_()
            launch()
            assert torch.equal(out, want), batch


def test_working_memory_goes_back_without_keys():
    """A caller of the drop-in alone holds no key set: what its call left in the
    library's pool goes back on request, and the next call takes it anew."""
    from tfhe_b200 import ops
    from tfhe_b200.engine import trim_working_memory
    four, rot = _dropin(3, 7, 3, n=240)
    scratch = four.numel() * 16
    a, lut = _draw((2, 240), 1).to(torch.float64), _draw((2, 2, 1024), 2).to(torch.float64)
    call = lambda: ops.multiply_seq_monomial(lut, a, four, 32, 7, 3, 1024, 3, rot, 1)
    want = call()
    torch.cuda.synchronize()
    kept = torch.cuda.mem_get_info()[0]
    trim_working_memory()
    assert torch.cuda.mem_get_info()[0] - kept >= scratch
    assert torch.equal(call(), want)


def test_forms_without_working_memory():
    """Calls at the limit of the device's memory: the key switch and packing make
    their digits in the kernel, the drop-in reads its key in place; the same words
    as with memory."""
    from tfhe_b200 import client64, lstm, ops, torus64
    from tfhe_b200.engine import launch_count, trim_working_memory
    rng = np.random.default_rng(0)
    words = lambda shape: rng.integers(0, 2 ** 32, size=shape, dtype=np.uint64).astype(np.uint32)
    keys = _keys(_params(1024, 120, 1, 9, 2))
    p64 = client64.Params64("ks64", N=1024, n=70, log2_beta_bs=13, l_bs=2, collapse=1, log2_beta_ks=4, l_ks=5,
                            sigma_glwe=2.0 ** 17, sigma_lwe=2.0 ** 40)
    keys64 = torus64.Keys64(client64.keygen(p64, 3))
    pack = lstm.PackingKey(words((1024, 4, 2, 1024)), 7, 4)
    pack64 = torus64.PackingKey64(rng.integers(0, 2 ** 63, size=(1024, 2, 2, 1024), dtype=np.uint64), 7, 2)
    four, rot = _dropin(3, 7, 3, n=240)
    B = 20000
    a, b = _draw((B, 1024), 1), _draw((B,), 2)
    a64, b64 = _draw((B, 1024), 3, torch.int64), _draw((B,), 4, torch.int64)
    idx, lut = torch.randint(0, 2048, (5, 80, 8), dtype=torch.int32, device="cuda"), _draw((5, 2, 1024), 5).to(torch.int64)
    bsk = four.reshape(2, 2, 3, 80, 8, 512).permute(3, 0, 2, 1, 4, 5).contiguous()
    import ctypes
    from tfhe_b200 import _lib
    out = torch.empty((5, 2, 1024), dtype=torch.int64, device="cuda")

    def dropin():
        ptr = lambda t: ctypes.c_void_p(t.data_ptr())
        _lib.check(_lib.load().tfhe_mul_bootstrap(
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), ptr(lut), lut.numel(), ptr(bsk),
            (ctypes.c_int64 * 6)(*bsk.shape), ptr(rot), 2048, ptr(idx), 7, 32, 3, 1024, ptr(out), 5))
        return out

    outs = [torch.empty((B, 120), dtype=torch.int32, device="cuda"), torch.empty((B,), dtype=torch.int32, device="cuda"),
            torch.empty((B, 70), dtype=torch.int64, device="cuda"), torch.empty((B,), dtype=torch.int64, device="cuda"),
            torch.empty((100, 2, 1024), dtype=torch.int32, device="cuda"),
            torch.empty((100, 2, 1024), dtype=torch.int64, device="cuda")]
    calls = [lambda: keys.keyswitch(a, b, outs[0], outs[1]), lambda: keys64.keyswitch(a64, b64, outs[2], outs[3], tensor_cores=1),
             lambda: pack.pack(a.view(100, 200, 1024), b.view(100, 200), out=outs[4]),
             lambda: pack64.pack(a64.view(100, 200, 1024), b64.view(100, 200), out=outs[5], tensor_cores=1), dropin]

    def run(call):
        before = launch_count()
        got = call()
        torch.cuda.synchronize()
        got = got if isinstance(got, tuple) else (got,)
        return [t.cpu() for t in got], launch_count() - before

    want = [run(call) for call in calls]
    trim_working_memory()
    hog = Hog(16 << 20)
    try:
        got = [run(call) for call in calls]
    finally:
        hog.close()
    for i, ((w, more), (g, launches)) in enumerate(zip(want, got)):
        assert launches < more, (i, launches, more)          # no digit matrix, no second layout
        assert all(torch.equal(x, y) for x, y in zip(w, g)), i


@pytest.mark.parametrize("shape", [(2048, 24, 2, 15, 2), (1024, 24, 3, 7, 3)])
def test_captured_bootstraps_replay_the_same_words(shape):
    """Every form of a degree inside a graph: new inputs in the captured buffers,
    the uncaptured call's words."""
    keys = _keys(_params(*shape))
    p = keys.params
    for batch in (1, 30, 60, 74, 148, 296, 600):
        a, b, lut = _draw((batch, p.N), 1), _draw((batch,), 2), _draw((batch, 2, p.N), 3)
        keys.pbs(a, b, lut)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = keys.pbs(a, b, lut)
        for seed in (4, 5):
            a.copy_(_draw((batch, p.N), seed))
            lut.copy_(_draw((batch, 2, p.N), seed + 9))
            graph.replay()
            want = keys.pbs(a, b, lut)
            assert torch.equal(out[0], want[0]) and torch.equal(out[1], want[1]), batch
        del graph


def test_two_streams_at_once():
    """Bootstraps, key switches, packing and traces whose kernels share the SMs
    (and their tensor memory) from two streams: each the words it has alone."""
    from tfhe_b200 import lstm, torus64
    rng = np.random.default_rng(1)
    words = lambda shape: rng.integers(0, 2 ** 32, size=shape, dtype=np.uint64).astype(np.uint32)
    keys = _keys(_params(2048, 24, 2, 15, 2))
    small = _keys(_params(1024, 24, 3, 7, 3))
    pack = lstm.PackingKey(words((1024, 4, 2, 1024)), 7, 4)
    galois = torus64.GaloisKeys64(rng.integers(0, 2 ** 63, size=(11, 5, 2, 2048), dtype=np.uint64), 8, 5)
    a, b, lut = _draw((700, 2048), 1), _draw((700,), 2), _draw((1, 2, 2048), 3)
    c, d, lut1 = _draw((40, 1024), 4), _draw((40,), 5), _draw((1, 2, 1024), 6)
    x, y = _draw((4, 128, 1024), 7), _draw((4, 128), 8)
    u, v = _draw((40, 2048), 9, torch.int64), _draw((40,), 10, torch.int64)
    first = lambda s=None: keys.pbs(a, b, lut, stream=s)
    second = lambda s=None: (*keys.keyswitch(a, b, stream=s), pack.pack(x, y, stream=s),
                             galois.pack_lwe_to_rlwe(u, v, stream=s), *small.pbs(c, d, lut1, stream=s))
    want = first(), second()
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    got = []
    for _ in range(5):
        with torch.cuda.stream(s1):
            one = first()
        with torch.cuda.stream(s2):
            two = [second() for _ in range(3)]
        got.append((one, two))
    torch.cuda.synchronize()
    for one, two in got:
        assert all(torch.equal(g, w) for g, w in zip(one, want[0]))
        for t in two:
            assert all(torch.equal(g, w) for g, w in zip(t, want[1]))
