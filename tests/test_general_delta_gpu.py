"""The generalised delta rule's kernels by themselves, against the recurrence in float64: prompts whose entries go in chunks of 16
tokens (heads of 64, 32 tokens an entry on average, one of 48 among more than two) and those next to that border, entries that end anywhere in a chunk, states that
are there already, decays next to one and far from it."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
SCALE, UNIT_EPS, EPS = 0.6065307, 1e-6, 1e-5


def problem(counts, heads, dim, rate, seed):
    rng = np.random.default_rng(seed)
    T, n = sum(counts), heads * dim
    f = lambda *s: rng.standard_normal(s).astype(np.float32)  # noqa: E731
    p = {"proj": f(T, 5 * n + 8), "x": f(T, n) * 2 + np.float32(rate), "w0": f(n), "a0": f(n), "gain": 1 + 0.1 * f(n), "state": f(len(counts), heads, dim, dim)}
    p["proj"][:, n:2 * n] *= 0.5
    if T > 20:                                              # keys that repeat: what one wrote is what the next takes off
        p["proj"][5:9, n:2 * n] = p["proj"][4, n:2 * n]
    return p


def exact(p, counts, heads, dim, unit_eps=UNIT_EPS):
    n = heads * dim
    sig = lambda z: 1 / (1 + np.exp(-z))  # noqa: E731
    q = {k: v.astype(np.float64) for k, v in p.items()}
    r, k, v, g, a = (q["proj"][:, i * n:(i + 1) * n].reshape(-1, heads, dim) for i in range(5))
    w = np.exp(-np.float64(np.float32(SCALE)) * sig(q["x"] + q["w0"])).reshape(-1, heads, dim)
    rate = sig(a + q["a0"].reshape(heads, dim))
    u = k / np.sqrt((k * k).sum(-1, keepdims=True) + unit_eps)
    out, state, at = np.zeros_like(v), np.zeros((len(counts), heads, dim, dim)), 0
    for s, c in enumerate(counts):
        S = q["state"][s].transpose(0, 2, 1).copy()             # the slot keeps [head, column, row]
        for t in range(at, at + c):
            held = np.einsum("hk,hkv->hv", u[t], S)
            S = w[t][..., None] * S - (rate[t] * u[t])[..., None] * held[:, None] + k[t][..., None] * v[t][:, None]
            out[t] = np.einsum("hk,hkv->hv", r[t], S)
        state[s], at = S.transpose(0, 2, 1), at + c
    y = out / np.sqrt((out * out).mean(-1, keepdims=True) + EPS) * q["gain"].reshape(heads, dim) * sig(g)
    return y.reshape(-1, n), state


def kernel(p, counts, heads, dim, lib=None, unit_eps=UNIT_EPS):
    import torch

    from easy_gpt.cpp_b200 import kernels

    lib = lib or kernels.library()
    fn = lib.eg_general_delta
    P, L, I, F = ctypes.c_void_p, ctypes.c_longlong, ctypes.c_int, ctypes.c_float
    fn.argtypes = [P, P, L] + [I] * 6 + [P, L, P, I, I] + [P] * 5 + [L, L, P, P, P, I, L, P] + [I] * 5 + [F] * 3 + [P]
    dev = {k: torch.from_numpy(v).cuda() for k, v in p.items()}
    T, n, slots = sum(counts), heads * dim, list(range(len(counts)))[::-1]
    state = torch.zeros(len(counts), heads * dim * dim, device="cuda")
    for s, slot in enumerate(slots):
        state[slot] = dev["state"][s].flatten()
    starts = torch.tensor(np.concatenate([[0], np.cumsum(counts)]), dtype=torch.int32, device="cuda")
    slot_ids = torch.tensor(slots, dtype=torch.int32, device="cuda")
    records = torch.full((T * heads * lib.eg_general_delta_record(dim),), float("nan"), device="cuda")
    y, o_raw = torch.full((T, n), float("nan"), device="cuda"), torch.full((T, n), float("nan"), device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    rc = fn(torch.cuda.current_stream().cuda_stream, dev["proj"].data_ptr(), dev["proj"].shape[1], 0, n, 2 * n, 3 * n, 4 * n, 5 * n, dev["x"].data_ptr(), n, None, 0, 8,
            dev["w0"].data_ptr(), dev["a0"].data_ptr(), dev["gain"].data_ptr(), records.data_ptr(), state.data_ptr(), n * dim, 0, starts.data_ptr(),
            slot_ids.data_ptr(), y.data_ptr(), 0, n, o_raw.data_ptr(), 4, T, len(counts), heads, dim, unit_eps, EPS, SCALE, status.data_ptr())
    torch.cuda.synchronize()
    assert rc == 0 and int(status[0]) == 0
    return y.cpu().numpy(), torch.stack([state[s] for s in slots]).reshape(len(counts), heads, dim, dim).cpu().numpy()


def off(got, want):
    return float(np.linalg.norm(got - want) / np.linalg.norm(want))


@pytest.mark.parametrize("rate", [-9.0, 0.0, 5.0])
@pytest.mark.parametrize("counts", [[32], [31], [33], [47, 17], [1, 63], [64, 1, 31], [257], [20, 12], [5, 90, 16, 48]])
@pytest.mark.parametrize("heads,dim", [(2, 64), (1, 64), (2, 48)])
def test_prompts_in_chunks(heads, dim, counts, rate):
    """Sums of 64 products and at most 16 factors in float32: 2^-24 times the root of some hundred roundings a token, which the
    decays and removals keep from adding up."""
    p = problem(counts, heads, dim, rate, len(counts) + 9 + int(rate) + counts[0])
    y, state = kernel(p, counts, heads, dim)
    want_y, want_state = exact(p, counts, heads, dim)
    assert np.isfinite(y).all()
    assert off(y, want_y) < 4e-6 and off(state, want_state) < 4e-6, (off(y, want_y), off(state, want_state))


@pytest.mark.parametrize("counts", [[33], [32], [47, 17], [5, 90, 16, 48]])
def test_keys_without_an_epsilon(counts):
    """unit_eps 0 is a key over its length: what fills up an entry's last chunk has no length, and must not divide by it."""
    p = problem(counts, 2, 64, 0.0, 77 + counts[0])
    y, state = kernel(p, counts, 2, 64, unit_eps=0.0)
    want_y, want_state = exact(p, counts, 2, 64, unit_eps=0.0)
    assert np.isfinite(y).all() and np.isfinite(state).all()
    assert off(y, want_y) < 4e-6 and off(state, want_state) < 4e-6


@pytest.mark.parametrize("rate, of_state, of_outputs", [(-9.0, 2.8e-7, 2.5e-7), (0.0, 8.8e-8, 1.5e-7), (5.0, 7.0e-8, 1.6e-7)])
@pytest.mark.parametrize("counts", [[257], [64], [40, 200]])
def test_errors_of_the_chunks(counts, rate, of_state, of_outputs):
    """A token at a time, S is rounded three times a token (2^-24 / sqrt(3) of its size each), and decays w forget: sqrt(3 / (1 - w^2)) of these at
    0 and 5.  The chunks are held to that; at -9, where nothing is forgotten, to what blocks of four tokens show (2.8e-7 at 257 tokens), and the
    outputs, which have roundings of their own (norm and gate), to what those show."""
    off_state, off_outputs = [], []
    for seed in range(4):
        p = problem(counts, 2, 64, rate, 100 + seed)
        y, state = kernel(p, counts, 2, 64)
        want_y, want_state = exact(p, counts, 2, 64)
        off_state.append(off(state, want_state))
        off_outputs.append(off(y, want_y))
    rms = lambda e: float(np.sqrt(np.mean(np.square(e))))  # noqa: E731
    assert rms(off_state) < of_state and rms(off_outputs) < of_outputs, (rms(off_state), rms(off_outputs))
