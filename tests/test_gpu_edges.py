"""Small parametrised tests at the sizes where a kernel's split or dispatch can go wrong
(edges of tiles, remainders, the smallest and largest of a range), against the CPU oracle."""
import numpy as np
import pytest

from helpers import BASE_SEED, check_close, from_dev, make_x, raw_weights, to_dev

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
