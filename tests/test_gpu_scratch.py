"""The scratch kept between calls: shared by the contexts of a device, still
there for one when another is gone, and given back when asked for."""
import numpy as np
import pytest

from conftest import pz, to_dev, to_host

pytestmark = pytest.mark.gpu


def test_scratch_outlives_a_context_and_is_given_back(gpu_available):
    import torch
    P = pz()
    g = np.random.default_rng(43)
    engines = [P.Engine("NI_2P") for _ in range(2)]
    p, N, Q = engines[0].p, engines[0].N, engines[0].Q
    ksk = g.integers(0, Q, (2 * p.ni_ks_d, N), dtype=np.uint64)
    keys = [e.upload_ni_ksk(ksk) for e in engines]
    rows = to_dev(g.integers(0, Q, (512, 2, N), dtype=np.uint64))
    out = torch.empty_like(rows)

    def switch(i):
        out.zero_()
        engines[i].ni_key_switch_device(keys[i], rows, out)
        torch.cuda.synchronize()
        return to_host(out)

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    want = switch(0)  # 512 x (0.8 MB of transformed digits + 64 KB of sums)
    kept = free()
    assert np.array_equal(switch(1), want)
    assert abs(free() - kept) < (64 << 20)  # the other context found it there
    keys[0].release()
    engines[0].close()
    assert np.array_equal(switch(1), want)
    assert free() > kept - (64 << 20)
    before = free()
    P.trim_scratch(0, keep=1 << 30)  # less than that is kept, or the rest goes
    assert free() >= before
    P.trim_scratch(0)
    assert free() - kept > (400 << 20)
    assert np.array_equal(switch(1), want)
    with pytest.raises(RuntimeError):
        P.trim_scratch(-1)
