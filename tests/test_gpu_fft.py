"""The FFT products at the edges of their exactness bound, and the forms of the
blind rotation at the batch sizes where one takes over from another."""
import numpy as np
import pytest

from conftest import oracle, oracle_setup, pz, to_dev, to_host

pytestmark = pytest.mark.gpu


def _extremes(Q):
    """Key words whose three 18-bit limbs are all as large as they get, and the
    ends of the centred range."""
    low = -((1 << 17) + (1 << 35) + (((1 << 17) - 1) << 36))  # limbs -2^17, -2^17, 1 - 2^17
    high = ((1 << 17) - 1) * (1 + (1 << 18) + (1 << 36))
    return [v % Q for v in (low, high, Q // 2, Q // 2 + 1, Q - 1, 0, 1 << 35, 1 << 17)]


@pytest.mark.parametrize("signs", ["same", "alternating", "random"])
def test_products_of_extreme_words(gpu_available, signs):
    """Digits of +-2^16 (products) and +-2^23 (automorphisms) in every coefficient
    against keys with every limb at its largest: the largest sums there are,
    exact word for word."""
    O = oracle()
    ev = O.Evaluator("NI_2P")
    i, N, Q = ev.info, ev.N, ev.Q
    g = np.random.default_rng(7)
    words = _extremes(Q)

    def pattern(v, shape):
        s = {"same": np.zeros(shape, bool), "alternating": np.arange(np.prod(shape)).reshape(shape) % 2 == 1,
             "random": g.integers(0, 2, shape).astype(bool)}[signs]
        return np.where(s, np.uint64((Q - v) % Q), np.uint64(v))

    rgsw = np.zeros((ev.n, i.rgsw_rows, N), np.uint64)
    autos = np.zeros((i.w + 1, i.auto_rows, N), np.uint64)
    for k, v in enumerate(words):
        rgsw[k] = pattern(v, rgsw[k].shape)
        autos[k] = pattern(v, autos[k].shape)
    ksk = np.zeros((i.lwe_d * N, ev.n + 1), np.uint64)
    okey = O.OracleKey(ev, O.ServerKeyCoeff(rgsw, autos, ksk))
    eng = pz().Engine("NI_2P")
    key = eng.upload_key(rgsw, autos, ksk)
    inputs = np.stack([pattern(v, (2, N)) for v in (Q // 2 - 1, Q // 2, Q // 2 + 1, (1 << 36) - 1, 1 << 36, 0)])
    idx = np.repeat(np.arange(len(words)), len(inputs)).astype(np.uint32)
    rl = np.concatenate([inputs] * len(words))
    for device, host in ((eng.rlwe_by_rgsw_device, okey.rlwe_by_rgsw), (eng.rlwe_auto_device, okey.rlwe_auto)):
        t = to_dev(rl)
        device(key, t, to_dev(idx))
        want = np.stack([host(r.reshape(-1), int(k)) for r, k in zip(rl, idx)])
        assert np.array_equal(to_host(t).reshape(len(rl), -1), want)


@pytest.mark.parametrize("param", ["I_2P_LB_SR", "NI_8P"])
def test_forms_agree(gpu_available, param):
    """The same key-switched ciphertexts in batches on either side of each form's
    range, with more ciphertexts than a form has places, and with few CTAs:
    the same words, and the oracle's for some."""
    import torch
    ev, _, coeff, okey = oracle_setup(param)
    eng = pz().Engine(param)
    key = eng.upload_key(coeff.rgsw, coeff.autos, coeff.ksk)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    most = 4 * sms + sms // 2 + 3
    r = oracle().Rng(b"\x5f" * 32)
    ks = r.uniform_mod(ev.info.lwe_q, most * (ev.n + 1)).reshape(most, -1).astype(np.uint32)
    gates = (np.arange(most) % 6).astype(np.uint8)

    def run(count, limit=0, split=-1):
        eng.set_split_threshold(split)
        eng.set_pbs_grid_limit(limit)
        out = to_dev(np.zeros((count, ev.L), np.uint64))
        eng.blind_rotate_device(key, to_dev(ks[:count]), to_dev(gates[:count]), out)
        return to_host(out)

    try:
        full = run(most)
        for count, limit, split in [(1, 0, -1), (sms // 2, 0, -1), (sms // 2 + 1, 0, -1), (sms, 0, 0), (sms + 1, 0, -1),
                                    (sms + sms // 2 + 1, 0, -1), (2 * sms + 1, 0, -1), (2 * sms + sms // 2 + 1, 0, -1),
                                    (4 * sms, 0, -1), (4 * sms + 3, 0, -1), (2 * sms + 1, sms + 1, -1),
                                    (13, 5, 74), (13, 5, 0), (2, 0, 0)]:
            assert np.array_equal(run(count, limit, split), full[:count]), (count, limit, split)
        # one gate through the debug entry point: the rotated RLWE is the oracle's
        c0 = r.uniform_mod(ev.Q, 2 * ev.L).reshape(2, ev.L)
        c1 = r.uniform_mod(ev.Q, 2 * ev.L).reshape(2, ev.L)
        out = to_dev(np.zeros((2, ev.L), np.uint64))
        eng.gate_batch_device(key, to_dev(gates[:2]), to_dev(c0), to_dev(c1), out)
        assert np.array_equal(to_host(out), okey.gate_batch(gates[:2], c0, c1, threads=2))
        assert eng.device_error() == 0
    finally:
        eng.set_split_threshold(-1)
        eng.set_pbs_grid_limit(0)


@pytest.mark.parametrize("count", [1, 3, 9, 287, 288, 290, 513])
def test_ni_key_switch_of_extreme_words(gpu_available, count):
    """Keys with both 27-bit limbs at their largest and values with as many
    non-zero digits as there can be, at counts around four rows to a warp and
    around a launch's largest batch."""
    O = oracle()
    ev = O.Evaluator("NI_8P")
    i, N, Q = ev.info, ev.N, ev.Q
    g = np.random.default_rng(11)
    low = -(1 << 26) - (((1 << 26) - 1) << 27)
    high = ((1 << 26) - 1) * (1 + (1 << 27))
    words = np.array([v % Q for v in (low, high, Q // 2, Q // 2 + 1, Q - 1, 1 << 26)], np.uint64)
    ksk = words[g.integers(0, len(words), (2 * i.ni_ks_d, N))]
    ksk[::3] = words[0]
    dense = ((1 << 50) - 1) // 3 << 3
    values = np.array([v % Q for v in (dense, -dense, dense << 1, Q // 2, Q // 2 + 1, 0, Q - 1)], np.uint64)
    rows = values[g.integers(0, len(values), (7, 2, N))]
    rows[0, 0] = values[0]
    rows[1, 0] = np.where(np.arange(N) % 2, values[0], values[1])
    want = np.stack([ev.ni_key_switch(ksk, r) for r in rows])
    pick = np.arange(count) % len(rows)
    eng = pz().Engine("NI_8P")
    d_out = to_dev(np.zeros((count, 2, N), np.uint64))
    eng.ni_key_switch_device(eng.upload_ni_ksk(ksk), to_dev(rows[pick]), d_out)
    assert np.array_equal(to_host(d_out).reshape(count, -1), want.reshape(len(rows), -1)[pick])


@pytest.mark.parametrize("shift", [0, 1])
def test_sample_extract_rows_off_16_bytes(gpu_available, shift):
    """Rows that start on and off a 16-byte boundary, runs that end in a launch's
    last CTA, RLWEs that change within a run, and an index past the batch."""
    eng = pz().Engine("NI_2P")
    N, Q, count = eng.N, eng.Q, 45
    g = np.random.default_rng(13)
    rl = g.integers(0, Q, (3, 2, N), dtype=np.uint64)
    idx = g.integers(0, 3 * N, count).astype(np.uint32)
    idx[:6] = [0, N - 1, N, 2 * N - 1, 2 * N, 3 * N - 1]
    idx[20] = 3 * N
    out = to_dev(np.full(shift + count * (N + 1), 5, np.uint64))
    eng.sample_extract_device(to_dev(rl), to_dev(idx), out[shift:])
    got = to_host(out)
    assert (got[:shift] == 5).all()
    for row, k in zip(got[shift:].reshape(count, N + 1), idx):
        if k >= 3 * N:
            assert (row == 5).all()
            continue
        a, b = rl[k // N]
        k = int(k) % N
        want = np.concatenate([b[k:k + 1], a[k::-1], np.uint64(Q) - a[:k:-1]])
        assert np.array_equal(row, want)


@pytest.mark.parametrize("pattern", ["zero", "same", "two", "spread"])
@pytest.mark.parametrize("param", ["I_2P_LB_SR", "NI_8P"])
def test_schedules_of_few_buckets(gpu_available, param, pattern):
    """Key switches whose LWEs put every index in one bucket (-g^0's or another),
    in two, or a few in many: windows from end to end, and the automorphisms
    before the first product."""
    O = oracle()
    ev = O.Evaluator(param)
    i, N, Q = ev.info, ev.N, ev.Q
    g = np.random.default_rng(17)
    rgsw = g.integers(0, Q, (ev.n, i.rgsw_rows, N), dtype=np.uint64)
    autos = g.integers(0, Q, (i.w + 1, i.auto_rows, N), dtype=np.uint64)
    col = np.arange(ev.n + 1)
    c = {"zero": 0 * col, "same": 1 + 0 * col, "two": np.where(col % 3 == 0, 1, i.lwe_q - 1), "spread": col}[pattern]
    ksk = np.broadcast_to(c.astype(np.uint64), (i.lwe_d * N, ev.n + 1)).copy()
    okey = O.OracleKey(ev, O.ServerKeyCoeff(rgsw, autos, ksk))
    eng = pz().Engine(param)
    key = eng.upload_key(rgsw, autos, ksk)
    gates = np.array([1, 4], np.uint8)
    c0, c1 = (g.integers(0, Q, (2, ev.L), dtype=np.uint64) for _ in range(2))
    out = to_dev(np.zeros((2, ev.L), np.uint64))
    eng.gate_batch_device(key, to_dev(gates), to_dev(c0), to_dev(c1), out)
    assert np.array_equal(to_host(out), okey.gate_batch(gates, c0, c1, threads=2))


@pytest.mark.parametrize("count, limit", [(1, 0), (3, 0), (7, 2)])
def test_waits_that_run_out_end_the_kernel(gpu_available, count, limit):
    """Two-CTA blind rotations whose waits all give up (one ciphertext per
    cluster, and several in turn): the kernel ends and says so in the error word,
    no copy or message of it disturbs what runs next, and with the usual limit
    the same call gives the one-CTA words."""
    eng = pz().Engine("I_2P_LB_SR")
    p = eng.p
    g = np.random.default_rng(23)
    key = eng.upload_key(g.integers(0, eng.Q, (p.lwe_n, p.rgsw_rows, eng.N), dtype=np.uint64),
                         g.integers(0, eng.Q, (p.n_auto_keys, p.auto_rows, eng.N), dtype=np.uint64),
                         g.integers(0, p.lwe_q, (p.lwe_d * eng.N, p.lwe_n + 1), dtype=np.uint64))
    c0, c1 = (to_dev(g.integers(0, eng.Q, (count, eng.L), dtype=np.uint64)) for _ in range(2))
    gates = to_dev((np.arange(count) % 6).astype(np.uint8))

    def run():
        out = to_dev(np.zeros((count, eng.L), np.uint64))
        eng.gate_batch_device(key, gates, c0, c1, out)
        return to_host(out)

    eng.set_split_threshold(0)
    want = run()
    eng.set_split_threshold(-1)
    eng.set_pbs_grid_limit(limit)
    for _ in range(2):
        eng.set_wait_limit(0)
        run()
        assert eng.device_error() == 1
        eng.set_wait_limit(-1)
        assert np.array_equal(run(), want)
        assert eng.device_error() == 0


def test_waits_that_run_out_are_errors_of_the_call(gpu_available):
    """What a synchronous call computed after a wait gave up is never returned as
    good: host-buffer gates, circuits and non-interactive inputs fail until the
    error word has been asked for, a server's step fails the jobs that it
    advanced and no others, and all of them work again afterwards."""
    P = pz()
    eng = P.Engine("NI_2P")
    p = eng.p
    g = np.random.default_rng(29)
    key = eng.upload_key(g.integers(0, eng.Q, (p.lwe_n, p.rgsw_rows, eng.N), dtype=np.uint64),
                         g.integers(0, eng.Q, (p.n_auto_keys, p.auto_rows, eng.N), dtype=np.uint64),
                         g.integers(0, p.lwe_q, (p.lwe_d * eng.N, p.lwe_n + 1), dtype=np.uint64))
    ksk = eng.upload_ni_ksk(g.integers(0, eng.Q, (2 * p.ni_ks_d, eng.N), dtype=np.uint64))
    C = P.Circuit()
    C.output(C.gate("nand", C.input(), C.input()))
    x = g.integers(0, eng.Q, (2, eng.L), dtype=np.uint64)
    b = g.integers(0, eng.Q, (1, eng.N), dtype=np.uint64)
    calls = [lambda: eng.gate_batch(key, np.array([1], np.uint8), x[:1], x[1:]), lambda: C.run(eng, key, x),
             lambda: eng.ni_ingest(ksk, b"\x05" * 32, b, 3)]
    want = [call() for call in calls]
    eng.set_wait_limit(0)
    S = P.Server(device=0, arena_bytes=1 << 22, max_items=64)
    sid = S.add_session(eng, key)
    for _ in range(2):
        for call in calls:  # the last has no such waits: it reports what the others set
            with pytest.raises(RuntimeError, match="gave up a wait"):
                call()
        assert eng.device_error() == 1
    wires = P.Circuit()
    wires.output(wires.input())  # no gate: nothing of it is computed
    job, other = S.submit(sid, C, x), S.submit(sid, wires, x[:1])
    with pytest.raises(RuntimeError, match="gave up a wait"):
        S.step()
    assert S.status(job)["state"] == P.server.FAILED and S.status(other)["state"] == P.server.DONE
    st = S.stats()
    assert (st["active"], st["failed"], st["done"], st["arena_slots_used"]) == (0, 1, 1, 0)
    assert np.array_equal(S.result(other), x[:1])
    assert eng.device_error() == 1
    eng.set_wait_limit(-1)
    for call, w in zip(calls, want):
        assert np.array_equal(call(), w)
    sid = S.add_session(eng, key)
    job = S.submit(sid, C, x)
    S.run_until_idle()
    assert np.array_equal(S.result(job), want[1])


@pytest.mark.parametrize("param", ["I_2P_LB_SR", "NI_8P"])
def test_resident_ciphertexts_of_each_shape(gpu_available, param):
    """The two-SM form holds a ciphertext per pair of SMs, the names of the other
    shape four per SM."""
    import torch
    eng = pz().Engine(param)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert [eng.pbs_slots(v) for v in range(5)] == [4 * sms, 4 * sms, 4 * sms, sms // 2, 4 * sms]


@pytest.mark.parametrize("count", [1, 147, 148, 149, 2961, 37887, 37888, 37893])
@pytest.mark.parametrize("order", ["in order", "shuffled", "runs"])
def test_sample_extract_of_many(gpu_available, order, count):
    """Batches around the distance at which CTAs take entries, and around the size
    from which they take several in a row (in order; shuffled; in runs of one RLWE
    with indices past the batch between them), against the definition."""
    import torch
    eng = pz().Engine("NI_2P")
    N, Q = eng.N, eng.Q
    g = np.random.default_rng(47)
    rl = to_dev(g.integers(0, Q, (6, 2, N), dtype=np.uint64))
    idx = np.arange(count) % (6 * N)
    if order == "shuffled":
        idx = g.permutation(6 * N)[idx]
    if order == "runs":
        idx = np.arange(count) // 5 % 6 * N + g.integers(0, N, count)
        idx[7::29], idx[8::40], idx[count - 1] = 6 * N, 6 * N + 3, 0xffffffff
    out = torch.full((count, N + 1), 5, dtype=torch.int64, device="cuda")
    eng.sample_extract_device(rl, to_dev(idx.astype(np.uint32)), out)
    col = torch.arange(N, device="cuda")
    for at in range(0, count, 1000):
        i = torch.from_numpy(idx[at:at + 1000].astype(np.int64)).cuda()
        there = i < 6 * N
        x, k = rl[torch.where(there, i // N, 0)], (i % N)[:, None]
        low = torch.gather(x[:, 0], 1, (k - col) % N)  # a_k .. a_0, then a_{N-1} .. a_{k+1}
        want = torch.cat([torch.gather(x[:, 1], 1, k), torch.where(col <= k, low, Q - low)], 1)
        assert torch.equal(out[at:at + 1000], torch.where(there[:, None], want, 5))


@pytest.mark.parametrize("width", [74, 149, 223, 297, 371, 595])
def test_circuit_levels_at_the_placing_boundaries(gpu_available, width):
    """A circuit's level gathers its inputs and scatters its outputs by wire; split
    over two launches, each half writes where the whole would have."""
    P = pz()
    eng = P.Engine("I_2P_LB_SR")
    p = eng.p
    g = np.random.default_rng(53)
    key = eng.upload_key(g.integers(0, eng.Q, (p.lwe_n, p.rgsw_rows, eng.N), dtype=np.uint64),
                         g.integers(0, eng.Q, (p.n_auto_keys, p.auto_rows, eng.N), dtype=np.uint64),
                         g.integers(0, p.lwe_q, (p.lwe_d * eng.N, p.lwe_n + 1), dtype=np.uint64))
    x = g.integers(0, eng.Q, (width + 1, eng.L), dtype=np.uint64)
    C = P.Circuit()
    wires = [C.input() for _ in x]
    gates = [C.gate(["and", "nand", "or", "nor", "xor", "xnor"][i % 6], wires[i], wires[i + 1]) for i in range(width)]
    C.outputs(gates[::-1])
    want = eng.gate_batch(key, (np.arange(width) % 6).astype(np.uint8), x[:-1], x[1:])
    assert np.array_equal(C.run(eng, key, x), want[::-1])
