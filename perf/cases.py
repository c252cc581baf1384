"""What this framework is timed on: the server-side work of FHE programs that
use its public entry points, from one gate to whole circuits of many sessions.

Every output is a whole number (ciphertext and key words modulo Q or q_ks),
computed exactly: two correct runs agree word for word.  Keys, ciphertexts and
shares are uniform words of the parameter set's shapes, which is how real ones
are distributed (each is masked by uniform words), so schedules and values are
those of real use.
"""
import importlib

import numpy as np
import torch

P = importlib.import_module("phantom-zone_b200")

DEVICE = "cuda"
SETS = ["I_2P_LB_SR", "I_4P", "I_8P", "NI_2P", "NI_4P_HB_FR", "NI_4P_LB_SR", "NI_8P"]
NI_SETS = SETS[3:]


def listed():
    return [
        # One gate per call: the plain form, a client-style loop of single bootstraps.
        {"name": "gate_1", "kind": "gates", "set": "I_2P_LB_SR", "count": 1},
        # A narrow level of a circuit: fewer gates than the GPU has SMs.
        {"name": "gates_37", "kind": "gates", "set": "NI_4P_LB_SR", "count": 37},
        # An ordinary batch, a little more than one wave of ciphertexts.
        {"name": "gates_500", "kind": "gates", "set": "I_4P", "count": 500},
        # A wide level of a wavefront, not a multiple of anything.
        {"name": "gates_2611", "kind": "gates", "set": "NI_8P", "count": 2611},
        # Ciphertexts that live on the host: copies in and out inside the call.
        {"name": "host_gates_129", "kind": "host_gates", "set": "I_8P", "count": 129},
        # One encrypted byte addition: a chain of narrow levels, latency throughout.
        {"name": "u8_add", "kind": "circuit", "set": "I_2P_LB_SR", "ops": "add", "copies": 1, "graph": False},
        # Many products and comparisons at once, captured once and replayed.
        {"name": "u8_wavefront", "kind": "circuit", "set": "NI_8P", "ops": "mul lt", "copies": 20, "graph": True},
        # Several users with keys of different parameter sets, served together.
        {"name": "sessions", "kind": "server", "sets": "I_2P_LB_SR I_4P I_8P", "jobs": 24, "ops": "add mul lt mux"},
        # RLWE x RGSW products by themselves: the kernel users build their own rotations from.
        {"name": "products_4096", "kind": "products", "set": "I_2P_LB_SR", "count": 4096},
        # Negacyclic transforms of a batch of polynomials, both directions.
        {"name": "ntt_4096", "kind": "ntt", "set": "NI_8P", "count": 4096},
        # A client's batch of non-interactive inputs: unseed, key switch, extract every bit.
        {"name": "ni_inputs_24", "kind": "ni_inputs", "set": "NI_8P", "count": 24},
        # The server key put together from the shares of all users, once per group of users.
        {"name": "ni_key_3_users", "kind": "ni_key", "set": "NI_4P_LB_SR", "users": 3},
    ]


def _log(rng, lo, hi):
    """A whole number in [lo, hi], spread evenly over its logarithm."""
    return min(hi, max(lo, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["gates", "gates", "gates", "host_gates", "circuit", "server", "products", "ntt", "ni_inputs"])
    if kind == "gates":
        return {"kind": kind, "set": rng.choice(SETS), "count": _log(rng, 1, 2600)}
    if kind == "host_gates":
        return {"kind": kind, "set": rng.choice(SETS), "count": _log(rng, 1, 900)}
    if kind == "circuit":
        ops = rng.sample(["add", "sub", "mul", "lt", "eq", "mux"], rng.randint(1, 3))
        return {"kind": kind, "set": rng.choice(SETS), "ops": " ".join(ops), "copies": _log(rng, 1, 12),
                "graph": rng.random() < 0.5}
    if kind == "server":
        return {"kind": kind, "sets": " ".join(rng.sample(SETS, rng.randint(1, 3))), "jobs": rng.randint(1, 20),
                "ops": " ".join(rng.sample(["add", "sub", "lt", "eq", "mux"], rng.randint(1, 3)))}
    if kind == "products":
        return {"kind": kind, "set": rng.choice(SETS), "count": _log(rng, 1, 6000)}
    if kind == "ntt":
        return {"kind": kind, "set": rng.choice(SETS), "count": _log(rng, 1, 6000)}
    return {"kind": kind, "set": rng.choice(NI_SETS), "count": _log(rng, 1, 48)}


# -- inputs -----------------------------------------------------------------------------
def _device_words(gen, bound, *shape):
    """Uniform words in [0, bound) on the device (u64 bits in an int64 tensor)."""
    return torch.randint(0, bound, shape, generator=gen, dtype=torch.int64, device=DEVICE)


def _seed32(rng):
    return rng.integers(0, 256, 32, dtype=np.uint8).tobytes()


def _engine_and_key(name, rng):
    """An engine and a server key uploaded in its seeded form, as a client sends it."""
    engine = P.Engine(name)
    p = engine.p
    rgsw = rng.integers(0, p.rlwe_q, (p.lwe_n, p.rgsw_rows, p.rlwe_n), dtype=np.uint64)
    auto_b = rng.integers(0, p.rlwe_q, (p.n_auto_keys, p.auto_d, p.rlwe_n), dtype=np.uint64)
    ksk_b = rng.integers(0, p.lwe_q, p.lwe_d * p.rlwe_n, dtype=np.uint64)
    return engine, engine.upload_key_seeded(rgsw, auto_b, _seed32(rng), ksk_b, _seed32(rng))


def _add_op(circuit, op):
    """One FheUint8 operation on fresh inputs, its results as outputs."""
    a, b = circuit.input_u8(), circuit.input_u8()
    if op in ("add", "sub", "mul"):
        circuit.outputs(getattr(circuit, "u8_" + op)(a, b))
    elif op in ("lt", "eq"):
        circuit.output(circuit.u8_cmp(op, a, b))
    else:
        circuit.outputs(circuit.u8_mux(a, b, circuit.input()))


def _circuit(ops, copies):
    circuit = P.Circuit()
    for _ in range(copies):
        for op in ops.split():
            _add_op(circuit, op)
    return circuit


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    state = dict(case)
    kind = case["kind"]
    if kind == "server":
        _prepare_server(state, case, rng, gen)
        return state
    if kind in ("ntt", "ni_inputs", "ni_key"):
        engine, key = P.Engine(case["set"]), None
    else:
        engine, key = _engine_and_key(case["set"], rng)
    p, q, n = engine.p, engine.Q, engine.N
    state.update(engine=engine, key=key)
    if kind == "gates":
        count = case["count"]
        state["gates"] = torch.randint(0, 6, (count,), generator=gen, dtype=torch.uint8, device=DEVICE)
        state["c0"] = _device_words(gen, q, count, engine.L)
        state["c1"] = _device_words(gen, q, count, engine.L)
        state["out"] = torch.empty_like(state["c0"])
    elif kind == "host_gates":
        count = case["count"]
        state["gates"] = rng.integers(0, 6, count, dtype=np.uint8)
        state["c0"] = rng.integers(0, q, (count, engine.L), dtype=np.uint64)
        state["c1"] = rng.integers(0, q, (count, engine.L), dtype=np.uint64)
    elif kind == "circuit":
        circuit = state["circuit"] = _circuit(case["ops"], case["copies"])
        state["inputs"] = _device_words(gen, q, circuit.n_inputs, engine.L)
        state["out"] = torch.empty((circuit.n_outputs, engine.L), dtype=torch.int64, device=DEVICE)
        if case["graph"]:
            state["stream"] = torch.cuda.Stream()
            state["stream"].wait_stream(torch.cuda.current_stream())
            circuit.capture_graph(engine, key, state["inputs"], state["out"], state["stream"])
    elif kind == "products":
        state["rlwe"] = _device_words(gen, q, case["count"], 2, n)
        state["index"] = torch.randint(0, p.lwe_n, (case["count"],), generator=gen, dtype=torch.int32, device=DEVICE)
    elif kind == "ntt":
        state["coefficients"] = _device_words(gen, q, case["count"], n)
        state["evaluations"] = _device_words(gen, q, case["count"], n)
    elif kind == "ni_inputs":
        count = case["count"]
        state["ksk"] = engine.upload_ni_ksk_seeded(rng.integers(0, q, (p.ni_ks_d, n), dtype=np.uint64), _seed32(rng))
        state["seed"] = _seed32(rng)
        state["b"] = _device_words(gen, q, count, n)
        state["index"] = torch.arange(count * n, dtype=torch.int32, device=DEVICE)
        state["seeded"] = torch.empty((count, 2, n), dtype=torch.int64, device=DEVICE)
        state["switched"] = torch.empty_like(state["seeded"])
        state["out"] = torch.empty((count * n, engine.L), dtype=torch.int64, device=DEVICE)
    else:
        _prepare_ni_key(state, case, rng, gen, engine)
    return state


def _prepare_server(state, case, rng, gen):
    sets = case["sets"].split()
    held = [_engine_and_key(name, rng) for name in sets]
    server = P.Server(device=0, arena_bytes=1 << 28, max_items=4096)
    sessions = [server.add_session(engine, key) for engine, key in held]
    circuits = [_circuit(op, 1) for op in case["ops"].split()]
    state.update(held=held, server=server, todo=[])
    for j in range(case["jobs"]):
        engine, circuit = held[j % len(held)][0], circuits[j % len(circuits)]
        state["todo"].append((sessions[j % len(held)], circuit,
                              _device_words(gen, engine.Q, circuit.n_inputs, engine.L),
                              torch.empty((circuit.n_outputs, engine.L), dtype=torch.int64, device=DEVICE)))


def _prepare_ni_key(state, case, rng, gen, engine):
    p, q, n, users = engine.p, engine.Q, engine.N, case["users"]
    per = -(-p.lwe_n // users)
    state["crs"] = _seed32(rng)
    state["shares"] = []
    for j in range(users):
        own = min(p.lwe_n, (j + 1) * per) - min(p.lwe_n, j * per)
        state["shares"].append({
            "ui_to_s_ksk": _device_words(gen, q, p.ni_ks_d, n),
            "ksk_zero_encs": _device_words(gen, q, users - 1, p.ni_ks_d, n),
            "self_leader_cts": _device_words(gen, q, own, max(p.rlrg_d_a, p.rlrg_d_b), n),
            "not_leader_cts": _device_words(gen, q, p.lwe_n - own, max(p.rgrg_d_a, p.rgrg_d_b), n),
            "rgsw_zero_encs": _device_words(gen, q, p.lwe_n, p.rgrg_d_a, n),
            "auto_keys": _device_words(gen, q, p.n_auto_keys, p.auto_d, n),
            "lwe_ksk": _device_words(gen, p.lwe_q, p.lwe_d * n),
        })
    new = lambda *shape: torch.empty(shape, dtype=torch.int64, device=DEVICE)  # noqa: E731
    state["out"] = (new(users, p.ni_ks_d, n), new(p.lwe_n, p.rgsw_rows, n), new(p.n_auto_keys, p.auto_d, n),
                    new(p.lwe_d * n))


# -- one pass ---------------------------------------------------------------------------
def run(state):
    kind = state["kind"]
    if kind == "server":
        return _run_server(state)
    engine, key = state["engine"], state["key"]
    if kind == "gates":
        engine.gate_batch_device(key, state["gates"], state["c0"], state["c1"], state["out"])
        return state["out"]
    if kind == "host_gates":
        return engine.gate_batch(key, state["gates"], state["c0"], state["c1"])
    if kind == "circuit":
        if state["graph"]:
            state["stream"].wait_stream(torch.cuda.current_stream())
            state["circuit"].replay_graph(state["stream"])
            torch.cuda.current_stream().wait_stream(state["stream"])
        else:
            state["circuit"].run_device(engine, key, state["inputs"], state["out"])
        return state["out"]
    if kind == "products":
        engine.rlwe_by_rgsw_device(key, state["rlwe"], state["index"])
        return state["rlwe"]
    if kind == "ntt":
        engine.ntt_forward_device(state["coefficients"])
        engine.ntt_backward_device(state["evaluations"])
        return state["coefficients"], state["evaluations"]
    if kind == "ni_inputs":
        engine.ni_unseed_device(state["seed"], state["b"], state["seeded"])
        engine.ni_key_switch_device(state["ksk"], state["seeded"], state["switched"])
        engine.sample_extract_device(state["switched"], state["index"], state["out"])
        return state["out"]
    engine.ni_aggregate_device(state["crs"], state["shares"], *state["out"])
    return state["out"]


def _run_server(state):
    server = state["server"]
    jobs = [server.submit(session, circuit, inputs, device_outputs=out)
            for session, circuit, inputs, out in state["todo"]]
    server.run_until_idle()
    for job in jobs:
        server.forget(job)
    return [out for _, _, _, out in state["todo"]]


# -- what a pass cannot do without ------------------------------------------------------
def _modmul_flops(polynomials, n):
    """Multiplications of polynomials' transforms: (N / 2) log2 N each, two operations a piece."""
    return polynomials * n * (n.bit_length() - 1)


def _bootstrap_work(p, count):
    """A blind rotation: per LWE coefficient two transforms in, two out and four
    pointwise products, and about as many automorphisms as nonempty windows
    (left out: they depend on the inputs).  Bytes: the server key once, the
    ciphertexts in and out."""
    n = p.rlwe_n
    key = p.lwe_n * p.rgsw_rows * n * 8 + p.n_auto_keys * p.auto_rows * n * 8 + p.lwe_d * n * (p.lwe_n + 1) * 4
    flops = count * (p.lwe_n * (_modmul_flops(4, n) + 8 * n) + 2 * p.lwe_d * n * (p.lwe_n + 1))
    return {"bytes": key + count * 3 * (n + 1) * 8, "flops": flops}


def work(case):
    kind = case["kind"]
    if kind == "server":
        sets, ops, jobs = case["sets"].split(), case["ops"].split(), case["jobs"]
        total = {"bytes": 0, "flops": 0}
        for i, name in enumerate(sets):
            gates = sum(_circuit(ops[j % len(ops)], 1).info()["gates"] for j in range(jobs) if j % len(sets) == i)
            part = _bootstrap_work(P.params(name), gates)
            total = {k: total[k] + part[k] for k in total}
        return total
    p = P.params(case["set"])
    n = p.rlwe_n
    if kind in ("gates", "host_gates"):
        return _bootstrap_work(p, case["count"])
    if kind == "circuit":
        return _bootstrap_work(p, _circuit(case["ops"], case["copies"]).info()["gates"])
    if kind == "products":
        key = min(case["count"], p.lwe_n) * p.rgsw_rows * n * 8
        return {"bytes": key + case["count"] * 4 * n * 8, "flops": case["count"] * (_modmul_flops(4, n) + 8 * n)}
    if kind == "ntt":
        return {"bytes": case["count"] * 4 * n * 8, "flops": _modmul_flops(2 * case["count"], n)}
    if kind == "ni_inputs":
        digits = case["count"] * p.ni_ks_d
        return {"bytes": p.ni_ks_d * 2 * n * 8 + case["count"] * n * 8 + case["count"] * n * (n + 1) * 8,
                "flops": _modmul_flops(digits + 2 * case["count"], n) + 4 * n * digits}
    users, d = case["users"], p.rgrg_d_a + p.rgrg_d_b
    share = (p.ni_ks_d * users + p.lwe_n * (p.rgrg_d_a + max(p.rgrg_d_a, p.rgrg_d_b))) * n * 8
    switched = p.lwe_n * d * p.ni_ks_d
    return {"bytes": users * share + p.lwe_n * p.rgsw_rows * n * 8,
            "flops": _modmul_flops(switched, n) + 4 * n * switched * users + _modmul_flops(2 * users * p.lwe_n * d, n)}


def exact(case, seed):
    """No output is a rounded number: all are whole words, equal between any two correct runs."""
    return None
