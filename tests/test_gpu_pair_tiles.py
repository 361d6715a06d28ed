"""tf_candidates_noalloc at the edges of its tiles (32 rows, 256 columns, 128 bodies in one CTA) against the pair
rules restated in numpy float32, which is exact: keys are integers and the comparisons' sums are rounded alike."""
import ctypes as C

import numpy as np
import pytest

from twofold_b200 import abi

F32 = np.float32


def _inputs(n, seed):
    rng = np.random.default_rng(seed)
    span = 0.8 * max(n, 2) ** (1.0 / 3.0)
    center = (rng.uniform(-0.5, 0.5, (n, 3)) * span).astype(F32)
    half = rng.uniform(0.1, 0.5, (n, 3)).astype(F32)
    grow = rng.uniform(0.0, 0.1, n).astype(F32)
    flags = rng.choice([7, 7, 7, 3, 1, 5, 0], n).astype(np.uint32)
    return center - half, center + half, grow, flags


def _overlap(lo_a, hi_a, lo_b, hi_b):
    return np.all((lo_a <= hi_b) & (lo_b <= hi_a), axis=-1)


def _expected(lo, hi, grow, flags):
    keys = []
    for a in range(len(grow) - 1):
        b = np.arange(a + 1, len(grow))
        either = flags[a] | flags[b]
        ok = ((flags[a] & flags[b] & abi.TF_PAIR_LIVE) != 0) & ((either & abi.TF_PAIR_DYNAMIC) != 0) & \
            ((either & abi.TF_PAIR_MOVING) != 0)
        reach = (grow[a] + grow[b])[:, None]
        ga, gb = grow[a], grow[b][:, None]
        ok &= _overlap(lo[a] - reach, hi[a] + reach, lo[b], hi[b])
        ok &= _overlap(lo[a], hi[a], lo[b] - reach, hi[b] + reach)
        ok &= _overlap(lo[a] - ga, hi[a] + ga, lo[b] - gb, hi[b] + gb)
        keys.append((np.uint64(a) << np.uint64(32)) | b[ok].astype(np.uint64))
    return np.concatenate(keys) if keys else np.zeros(0, np.uint64)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [0, 1, 2, 31, 32, 33, 127, 128, 129, 160, 255, 256, 257, 289, 1000, 4065, 4096])
def test_pairs_at_the_edges_of_the_tiles(n):
    torch = pytest.importorskip("torch")
    lib = abi.load()
    lo, hi, grow, flags = _inputs(n, 7 + n)
    expected = _expected(lo, hi, grow, flags)
    dev = [torch.from_numpy(np.ascontiguousarray(x).view(np.int32) if x.dtype == np.uint32 else np.ascontiguousarray(x)).to("cuda")
           for x in (lo.reshape(-1), hi.reshape(-1), grow, flags)]
    for capacity in (len(expected) + 5, max(len(expected) - 3, 0)):
        keys = torch.full((max(capacity, 1),), -1, dtype=torch.int64, device="cuda")
        count = torch.full((1,), -7, dtype=torch.int32, device="cuda")
        abi.check(lib.tf_candidates_noalloc(*(x.data_ptr() for x in dev), n, keys.data_ptr(), capacity, count.data_ptr(),
                                            C.c_void_p(torch.cuda.current_stream().cuda_stream)), lib)
        got = keys.cpu().numpy().view(np.uint64)
        assert int(count.item()) == len(expected)
        kept = min(capacity, len(expected))
        assert np.array_equal(got[:kept], expected[:kept])
        assert np.all(got[kept:] == np.uint64(0xFFFFFFFFFFFFFFFF)), "keys past the count or the capacity were written"
