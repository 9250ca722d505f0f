"""Small parametrised tests at the sizes where a kernel's split or dispatch can go wrong
(edges of tiles, remainders, the smallest and largest of a range), against the CPU oracle."""
import numpy as np
import pytest

from helpers import BASE_SEED, _ordinal, check_close, from_dev, make_x, raw_weights, to_dev

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    import torch
    import cudalm_agent_b200 as eng
    assert torch.cuda.is_available()
    eng.load_library()
    yield eng
    assert eng.device_status() == 0, "a device-side wait ran out during the tests"


@pytest.mark.parametrize("k", [1, 2, 8, 31, 32, 33, 50, 63, 64])
def test_sampling_at_every_share_of_a_warp(eng, orc, k):
    """One to 64 candidates (two per lane), few and many kept by top-p, flat and peaked
    lists, more rows than a block: tokens and generator states equal the oracle's."""
    import torch
    rng = np.random.default_rng(BASE_SEED + k)
    M, n = 37, 64
    idx = np.stack([rng.permutation(248320)[:n] for _ in range(M)]).astype(np.int32)
    spread = np.where(np.arange(M) % 3 == 0, 0.0, np.where(np.arange(M) % 3 == 1, 1.0, 8.0))
    val = -np.sort(-rng.standard_normal((M, n)) * spread[:, None], axis=1)
    val = orc.f32_to_bf16_bits(np.ascontiguousarray(val, np.float32))
    state0 = rng.integers(0, 2 ** 62, M).astype(np.uint64)
    for t, p in ((0.8, 0.95), (1.3, 1.0), (0.05, 0.5), (2.0, 1e-6)):
        st = torch.from_numpy(state0.astype(np.int64)).cuda()
        got = from_dev(eng.sample_topk(to_dev(idx), to_dev(val, torch.bfloat16), float(np.float32(t)), k,
                                       float(np.float32(p)), st))
        new = st.cpu().numpy().astype(np.uint64)
        for m in range(M):
            want, state = orc.sample_from_topk(idx[m], val[m], float(np.float32(t)), k,
                                               float(np.float32(p)), int(state0[m]))
            assert (got[m], int(new[m])) == (want, state), (m, t, p)


def _quantize_equal(eng, orc, wb):
    import torch
    packed, scale = eng.quantize_w4a16(to_dev(wb, torch.bfloat16))
    want_p, want_s = orc.quantize_w4a16(wb)
    assert np.array_equal(from_dev(packed), want_p)
    assert np.array_equal(from_dev(scale).view(np.uint16), want_s.view(np.uint16))


def test_quantizer_on_every_pair_of_significands(eng, orc):
    """The group maximum takes each of the 128 bf16 significands, the other values of its
    groups every bf16 of the same and the next 13 lower exponents, of either sign: each
    rounding boundary and each exact tie there is (14 |w| an odd multiple of the maximum)."""
    rest = np.arange((127 - 13) << 7, (127 << 7) + 128, dtype=np.uint16)
    groups = []
    for a in range(128):
        top = (127 << 7) | a
        w = rest[rest <= top]
        w = np.concatenate([w, w | 0x8000])
        w = np.concatenate([w, np.zeros(-w.size % 127, np.uint16)]).reshape(-1, 127)
        groups.append(np.concatenate([np.full((w.shape[0], 1), top, np.uint16), w], axis=1))
    wb = np.concatenate(groups)
    n = wb.shape[0] // 8
    _quantize_equal(eng, orc, np.ascontiguousarray(wb[:n * 8].reshape(n, 1024)))


@pytest.mark.parametrize("exponent", [1, 20, 34, 36, 38, 40, 127, 216, 218, 220, 222, 250, 254])
def test_quantizer_over_the_exponents(eng, orc, exponent):
    """Scales either side of the range in which the packed arithmetic is exact, down to
    subnormal ones and up to the largest bf16."""
    rng = np.random.default_rng(BASE_SEED + exponent)
    e = np.clip(exponent - rng.integers(0, 10, (64, 256)), 0, 254).astype(np.uint16)
    wb = (e << 7) | rng.integers(0, 128, e.shape, dtype=np.uint16) | (rng.integers(0, 2, e.shape, dtype=np.uint16) << 15)
    _quantize_equal(eng, orc, wb.astype(np.uint16))


@pytest.mark.parametrize("N,K", [(1, 128), (1, 1920), (1, 2048), (1, 2176), (15, 128), (17, 128), (129, 384),
                                 (4737, 1024), (18944, 128), (18945, 128)])
def test_quantizer_group_counts(eng, orc, N, K):
    """Group counts around a warp's sixteen and around a whole grid of them."""
    rng = np.random.default_rng(BASE_SEED + N)
    _quantize_equal(eng, orc, orc.f32_to_bf16_bits((rng.standard_normal((N, K)) * 0.02).astype(np.float32)))


# the many-row kernel (also from 17 rows): activation tiles of 64 (few units), 128 and 256 rows; tile remainders of
# either side; one group, an odd number of groups and more groups than any ring holds
ROWS_SHAPES = [(304, 1024, 17), (1104, 2048, 40), (136, 384, 64), (1, 128, 65), (63, 128, 129), (64, 256, 127), (127, 384, 128), (129, 2944, 66),
               (513, 4608, 96), (1023, 256, 2048), (1024, 384, 2047), (4100, 128, 2085), (4224, 640, 1793),
               (19000, 128, 70), (40000, 128, 33)]


@pytest.fixture
def no_lean(eng):
    prev = eng.set_direct_path_max_bytes(0)
    yield
    eng.set_direct_path_max_bytes(prev)


@pytest.mark.parametrize("N,K,M", ROWS_SHAPES)
def test_many_rows(eng, orc, no_lean, N, K, M):
    """Plain, residual (also in place) and gate/up forms of many rows against the oracle,
    and twice for equal bits; outputs off 16 bytes and off the matrix stay untouched."""
    import torch
    W, S = raw_weights(N, K, BASE_SEED + N)
    x = make_x(orc, (M, K), BASE_SEED + M, "outlier")
    want = orc.batch_gemv_bf16(W, S, x, threads=8)
    Wd, Sd, xd = to_dev(W), to_dev(S, torch.float16), to_dev(x, torch.bfloat16)
    buf = torch.full((M * N + 3,), 7.0, device="cuda", dtype=torch.bfloat16)
    y = buf[1:1 + M * N].view(M, N)
    got = from_dev(eng.batch_int4_gemv_bf16(Wd, Sd, xd, y))
    check_close(orc, got, want, f"{N}x{K} M={M}")
    assert buf[0] == 7.0 and bool((buf[1 + M * N:] == 7.0).all())
    assert np.array_equal(got, from_dev(eng.batch_int4_gemv_bf16(Wd, Sd, xd)))

    lin = eng.W4A16Linear(Wd, Sd)
    res = make_x(orc, (M, N), BASE_SEED + 1)
    h = to_dev(res, torch.bfloat16)
    want_res = orc.add_bf16(res.ravel(), got.ravel()).reshape(M, N)
    assert np.array_equal(from_dev(eng.linear_residual_bf16(lin, xd, h)), want_res)
    assert np.array_equal(from_dev(eng.linear_residual_bf16(lin, xd, h, y=h)), want_res)

    W2, S2 = raw_weights(N, K, BASE_SEED + N + 1)
    up = eng.W4A16Linear(to_dev(W2), to_dev(S2, torch.float16))
    g_y, u_y = eng.gate_up_bf16(lin, up, xd)
    assert np.array_equal(from_dev(g_y), got)
    fused = from_dev(eng.gate_up_silu_bf16(lin, up, xd))
    two = orc.silu_mul_bf16(from_dev(g_y).ravel(), from_dev(u_y).ravel()).reshape(M, N)
    off = _ordinal(fused) - _ordinal(two)
    assert np.abs(off).max() <= 1 and np.count_nonzero(off) <= max(2, 2e-3 * off.size)


def test_many_rows_in_one_call_with_few(eng, orc):
    """linear_multi over projections of different shapes and row counts, some below 65 rows."""
    import torch
    items, want = [], []
    for i, (N, K, M) in enumerate([(300, 384, 200), (16, 1024, 3), (1000, 128, 65), (129, 256, 500)]):
        W, S = raw_weights(N, K, BASE_SEED + i)
        x = make_x(orc, (M, K), BASE_SEED + i)
        want.append(orc.batch_gemv_bf16(W, S, x, threads=8))
        items.append((eng.W4A16Linear(to_dev(W), to_dev(S, torch.float16)), to_dev(x, torch.bfloat16),
                      torch.empty((M, N), device="cuda", dtype=torch.bfloat16)))
    eng.linear_multi(items)
    for (_, _, y), w in zip(items, want):
        check_close(orc, from_dev(y), w)


@pytest.mark.parametrize("N,K,M", [(1, 128, 9), (17, 384, 16), (40, 1152, 10), (5003, 2944, 13), (1000, 1024, 15),
                                   (33, 4224, 1), (100, 8192, 8), (257, 8320, 16), (15, 16384, 9), (700, 4096, 12),
                                   (100, 4224, 17), (257, 2176, 33), (2368, 2176, 64), (17, 8192, 40), (1024, 3584, 32),
                                   (512, 2048, 48), (2368, 2048, 49), (1, 2176, 64)])
def test_lean_kernel_on_more_rows_and_any_k(eng, orc, N, K, M):
    """One, two, four, six and eight column tiles, K splits of equal and unequal length, K beyond the
    streaming kernel's limit: plain, residual and gate/up forms against the oracle."""
    import torch
    W, S = raw_weights(N, K, BASE_SEED + N)
    W2, S2 = raw_weights(N, K, BASE_SEED + N + 1)
    x = make_x(orc, (M, K), BASE_SEED + M, "outlier")
    res = make_x(orc, (M, N), BASE_SEED + 1)
    want = orc.batch_gemv_bf16(W, S, x, threads=8)
    lin, up = (eng.W4A16Linear(to_dev(w), to_dev(s, torch.float16)) for w, s in ((W, S), (W2, S2)))
    xd = to_dev(x, torch.bfloat16)
    prev = eng.set_direct_path_max_bytes(1 << 40)
    try:
        got = from_dev(eng.batch_int4_gemv_bf16(lin.weight, lin.scale, xd))
        other = from_dev(eng.batch_int4_gemv_bf16(up.weight, up.scale, xd))
        added = from_dev(eng.linear_residual_bf16(lin, xd, to_dev(res, torch.bfloat16)))
        fused = from_dev(eng.gate_up_silu_bf16(lin, up, xd))
        for m in {0, M // 2, M - 1} if M <= 16 else ():  # a row's bits do not depend on its batch
            assert np.array_equal(from_dev(eng.int4_gemv_bf16(lin.weight, lin.scale, xd[m].contiguous())), got[m])
    finally:
        eng.set_direct_path_max_bytes(prev)
    check_close(orc, got, want, f"{N}x{K} M={M}")
    assert np.array_equal(added, orc.add_bf16(res.ravel(), got.ravel()).reshape(M, N))
    two = orc.silu_mul_bf16(got.ravel(), other.ravel()).reshape(M, N)
    off = _ordinal(fused) - _ordinal(two)
    assert np.abs(off).max() <= 1 and np.count_nonzero(off) <= max(2, 2e-3 * off.size)


def test_bound_calls_take_and_refuse_what_the_checks_do(eng):
    """The compiled binding answers exactly the calls the Python checks would pass on, and
    leaves the rest to them: the same bits through either, the same errors as without it."""
    import torch
    from cudalm_agent_b200 import api
    W, S = raw_weights(64, 256, BASE_SEED)
    W2, S2 = raw_weights(64, 256, BASE_SEED + 1)
    l1, l2 = (eng.W4A16Linear(to_dev(w), to_dev(s, torch.float16)) for w, s in ((W, S), (W2, S2)))
    x = torch.randn(5, 256, device="cuda").bfloat16()
    res, y = torch.randn(5, 64, device="cuda").bfloat16(), torch.empty(5, 64, device="cuda", dtype=torch.bfloat16)
    calls = [
        lambda x, y: eng.int4_gemv_bf16(l1.weight, l1.scale, x[0], y[0]),
        lambda x, y: eng.batch_int4_gemv_bf16(l1.weight, l1.scale, x, y),
        lambda x, y: eng.linear_multi([(l1, x, y)]),
        lambda x, y: eng.gate_up_silu_bf16(l1, l2, x, y),
        lambda x, y: eng.linear_residual_bf16(l1, x, res, y),
    ]
    native = api._native

    class Off:
        def __getattr__(self, name):
            return lambda *a: -1

    for i, call in enumerate(calls):
        out = []
        for binding in (native, Off()):
            api._native = binding
            try:
                y.zero_()
                call(x, y)
                out.append(from_dev(y).copy())
                for bad_x, bad_y in ((x.float(), y), (x.cpu(), y), (x, y.float()), (x.t().contiguous().t(), y)):
                    if i > 2 and bad_y is not y:
                        continue  # these two take the output as it is
                    with pytest.raises(ValueError):
                        call(bad_x, bad_y)
                if i in (0, 1):
                    with pytest.raises(ValueError):
                        call(x[:, :128].contiguous(), y)
            finally:
                api._native = native
        assert np.array_equal(out[0], out[1]), i
    assert native.batch(l1.weight, l1.scale, x, y) == 0
    assert native.batch(l1.weight, l1.scale, x.t().contiguous().t(), y) == -1
    assert native.batch(l1.weight, l1.scale, x, y[:, :32]) == -1
    assert native.linear_residual(l1, x, res[:, :63], y) == -1
    assert native.gate_up_silu(l1, None, x, y) == -1
    assert native.multi([(l1, x, y)] * 5) == -1 and native.multi([]) == -1
    seen = []  # a wrapped tensor is not taken
    torch.func.vmap(lambda v: seen.append(native.gemv(l1.weight, l1.scale, v, y[0])) or v)(x)
    assert seen == [-1]
    torch.cuda.synchronize()


def test_many_row_silu_on_every_bf16_value(eng, orc):
    """The many-row kernel's silu corrects an approximate quotient: every bf16 gate value gives
    the bits of the lean kernel, which divides with correct rounding."""
    import torch
    W = np.zeros((8, 64), np.uint8)
    W[:, 0] = 0x01                       # the gate output is x[0] ...
    W2 = np.zeros((8, 64), np.uint8)
    W2[:, 0] = 0x10                      # ... and the up output x[1]
    one = np.full((8, 1), 0x3C00, np.uint16)
    gate, up = (eng.W4A16Linear(to_dev(w), to_dev(one, torch.float16)) for w in (W, W2))
    bits = np.arange(65536, dtype=np.uint16)
    finite = bits[(bits & 0x7F80) != 0x7F80]  # an infinity times a weight of zero is a NaN
    x = np.zeros((finite.size, 128), np.uint16)
    x[:, 0], x[:, 1] = finite, 0x3F80
    xd = to_dev(x, torch.bfloat16)
    got = eng.gate_up_silu_bf16(gate, up, xd)
    want = torch.cat([eng.gate_up_silu_bf16(gate, up, xd[i:i + 8]) for i in range(0, finite.size, 8)])
    assert np.array_equal(from_dev(got), from_dev(want))
