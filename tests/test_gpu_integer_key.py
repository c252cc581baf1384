"""Keys without their FFT form (asked for, or for lack of device memory): the
integer kernels of the N = 2048 one-digit sets, against the oracle and against
the FFT kernels."""
import numpy as np
import pytest

from conftest import oracle, oracle_setup, pz, to_dev, to_host

pytestmark = pytest.mark.gpu


def _both(eng, rgsw, autos, ksk):
    """The same key with and without its FFT form."""
    fast = eng.upload_key(rgsw, autos, ksk)
    eng.set_key_fft(False)
    slow = eng.upload_key(rgsw, autos, ksk)
    eng.set_key_fft(True)
    assert fast.has_fft and not slow.has_fft
    return fast, slow


@pytest.mark.parametrize("param", ["I_2P_LB_SR", "NI_8P"])
def test_gates_and_rotations(gpu_available, param):
    """Gate batches word for word the oracle's; blind rotations of odd counts,
    with as many CTAs as ciphertexts and with few, those of the FFT form; the
    exported blob is the same and imports either way."""
    ev, _, coeff, okey = oracle_setup(param)
    eng = pz().Engine(param)
    fast, slow = _both(eng, coeff.rgsw, coeff.autos, coeff.ksk)
    assert slow.device_bytes < fast.device_bytes
    r = oracle().Rng(b"\x3c" * 32)
    c0, c1 = (r.uniform_mod(ev.Q, 6 * ev.L).reshape(6, ev.L) for _ in range(2))
    gates = np.arange(6, dtype=np.uint8)
    assert np.array_equal(eng.gate_batch(slow, gates, c0, c1), okey.gate_batch(gates, c0, c1, threads=6))
    ks = r.uniform_mod(ev.info.lwe_q, 451 * (ev.n + 1)).reshape(451, -1).astype(np.uint32)

    def rotate(key, count, limit=0):
        eng.set_pbs_grid_limit(limit)
        out = to_dev(np.zeros((count, ev.L), np.uint64))
        eng.blind_rotate_device(key, to_dev(ks[:count]), to_dev((np.arange(count) % 6).astype(np.uint8)), out)
        eng.set_pbs_grid_limit(0)
        return to_host(out)

    want = rotate(fast, 451)
    for count, limit in [(1, 0), (74, 0), (75, 0), (296, 0), (297, 0), (451, 0), (13, 3), (90, 5)]:  # to 74 on two SMs each
        assert np.array_equal(rotate(slow, count, limit), want[:count]), (count, limit)
    blob = slow.export()
    assert blob == fast.export()
    eng.set_key_fft(False)
    again = eng.import_key(blob)
    eng.set_key_fft(True)
    assert not again.has_fft and again.device_bytes == slow.device_bytes and eng.import_key(blob).has_fft
    assert np.array_equal(rotate(again, 3), want[:3])


@pytest.mark.parametrize("pattern", ["zero", "two", "spread"])
def test_schedules_of_few_buckets(gpu_available, pattern):
    """Windows from end to end and automorphisms before the first product."""
    O = oracle()
    ev = O.Evaluator("I_2P_LB_SR")
    i, N, Q = ev.info, ev.N, ev.Q
    g = np.random.default_rng(31)
    rgsw = g.integers(0, Q, (ev.n, i.rgsw_rows, N), dtype=np.uint64)
    autos = g.integers(0, Q, (i.w + 1, i.auto_rows, N), dtype=np.uint64)
    col = np.arange(ev.n + 1)
    c = {"zero": 0 * col, "two": np.where(col % 3 == 0, 1, i.lwe_q - 1), "spread": col}[pattern]
    ksk = np.broadcast_to(c.astype(np.uint64), (i.lwe_d * N, ev.n + 1)).copy()
    okey = O.OracleKey(ev, O.ServerKeyCoeff(rgsw, autos, ksk))
    eng = pz().Engine("I_2P_LB_SR")
    _, slow = _both(eng, rgsw, autos, ksk)
    gates = np.array([1, 4], np.uint8)
    c0, c1 = (g.integers(0, Q, (2, ev.L), dtype=np.uint64) for _ in range(2))
    assert np.array_equal(eng.gate_batch(slow, gates, c0, c1), okey.gate_batch(gates, c0, c1, threads=2))


def test_products_and_automorphisms(gpu_available):
    """RLWE x RGSW products (general and trivial) and automorphisms by themselves,
    every slot, inputs at the ends of the centred range, an index past the keys."""
    ev, _, coeff, okey = oracle_setup("NI_2P")
    eng = pz().Engine("NI_2P")
    fast, slow = _both(eng, coeff.rgsw, coeff.autos, coeff.ksk)
    w, n, Q = eng.p.w, eng.p.lwe_n, eng.Q
    g = np.random.default_rng(37)
    rl = g.integers(0, Q, (w + 3, 2, eng.N), dtype=np.uint64)
    rl[0], rl[1, 0], rl[1, 1], rl[2] = 0, Q - 1, Q // 2, Q // 2 + 1
    index = g.integers(0, n, w + 3).astype(np.uint32)
    slot = np.arange(w + 3, dtype=np.uint32) % (w + 1)
    for call, host, idx, end in ((eng.rlwe_by_rgsw_device, okey.rlwe_by_rgsw, index, n),
                                 (eng.rlwe_auto_device, okey.rlwe_auto, slot, w + 1)):
        idx[-1] = end
        out = []
        for key in (fast, slow):
            t = to_dev(rl)
            call(key, t, to_dev(idx))
            out.append(to_host(t).reshape(len(rl), -1))
        assert np.array_equal(out[0], out[1])
        want = [host(x.reshape(-1), int(k)) for x, k in zip(rl[:4], idx[:4])]
        assert np.array_equal(out[1][:4], np.stack(want))
        assert np.array_equal(out[1][-1], rl[-1].reshape(-1))
        trivial = []
        for key in (fast, slow):
            t = to_dev(rl)
            call(key, t, to_dev(idx), trivial=True)
            trivial.append(to_host(t))
        assert np.array_equal(trivial[0], trivial[1])


@pytest.mark.parametrize("width", [5, 75, 149, 223, 297, 371, 596])
def test_server_with_keys_of_both_forms(gpu_available, width):
    """A step whose width lies on either side of each placing boundary (the ragged
    launches scatter their outputs): sessions whose keys have the FFT form run over
    it in a launch of their own beside one whose key does not, every job with the
    words it has alone."""
    P = pz()
    g = np.random.default_rng(41)
    sessions = []
    S = P.Server(device=0, arena_bytes=1 << 27, max_items=4096)
    for param, fft in (("I_2P_LB_SR", True), ("NI_8P", True), ("I_8P", False)):
        eng = P.Engine(param)
        p = eng.p
        eng.set_key_fft(fft)
        key = eng.upload_key(g.integers(0, eng.Q, (p.lwe_n, p.rgsw_rows, eng.N), dtype=np.uint64),
                             g.integers(0, eng.Q, (p.n_auto_keys, p.auto_rows, eng.N), dtype=np.uint64),
                             g.integers(0, p.lwe_q, (p.lwe_d * eng.N, p.lwe_n + 1), dtype=np.uint64))
        assert key.has_fft == fft
        sessions.append((eng, key, S.add_session(eng, key)))
    counts = (width // 2, width - width // 2, 3)
    jobs = []
    for (eng, key, sid), count in zip(sessions, counts):
        gates = (np.arange(count) % 6).astype(np.uint8)
        C = P.Circuit()
        inputs = [C.input() for _ in range(count + 1)]
        C.outputs([C.gate(["and", "nand", "or", "nor", "xor", "xnor"][t], inputs[i], inputs[i + 1])
                   for i, t in enumerate(gates)])
        x = g.integers(0, eng.Q, (count + 1, eng.L), dtype=np.uint64)
        jobs.append((S.submit(sid, C, x), eng.gate_batch(key, gates, x[:-1], x[1:])))
    assert S.step() == width + 3
    st = S.stats()
    assert st["done"] == 3 and st["launches"] == 4  # a key switch and a blind rotation for either form
    for job, want in jobs:
        assert np.array_equal(S.result(job), want)
