"""The delta rule by chunks of 64 tokens against the recurrence in double, token by token: outputs
and the state left behind, at the edges of chunks, head sizes and column blocks."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def rounded(array):
    return torch.tensor(np.asarray(array), dtype=torch.float32).to(torch.bfloat16).cuda()


def plain(q, k, v, beta, log_decay, state):
    """``q, k [T, H, D]``, ``v [T, H, V]``, state ``[H, D, V]``, all double."""
    out = np.zeros((q.shape[0], q.shape[1], v.shape[2]))
    for t in range(q.shape[0]):
        state = np.exp(log_decay[t])[:, None, None] * state
        u = beta[t][:, None] * (v[t] - np.einsum("hdv,hd->hv", state, k[t]))
        state = state + k[t][:, :, None] * u[:, None]
        out[t] = np.einsum("hdv,hd->hv", state, q[t])
    return out, state


def packed_state(state, per_head):
    """``[H, D, V]`` as a request's state row keeps it: [row % 16][column][row / 16]."""
    heads, dim, vdim = state.shape
    parts = per_head // (16 * vdim)
    wide = np.zeros((heads, 16 * parts, vdim))
    wide[:, :dim] = state
    return wide.reshape(heads, parts, 16, vdim).transpose(0, 2, 3, 1).reshape(heads, -1)


@pytest.mark.parametrize("unit", [True, False])
@pytest.mark.parametrize("heads,qk_heads,dim,vdim,lengths", [
    (4, 2, 128, 128, (64, 1, 129)),        # whole chunks, a single token, one token over
    (2, 2, 120, 136, (65, 63)),            # padded keys, a second block of columns
    (3, 1, 48, 40, (200,)),
    (2, 1, 8, 8, (1, 16, 17, 2)),          # the smallest heads
    (40, 40, 64, 128, (3, 70, 1, 5)),      # more blocks than SMs: eight warps of columns
])
def test_chunks_against_the_recurrence(heads, qk_heads, dim, vdim, lengths, unit):
    from helix_runtime_b200.ops import library as ops
    rng = np.random.default_rng(dim + vdim + unit)
    tokens = sum(lengths)
    q, k = (rounded(rng.normal(size=(tokens, qk_heads * dim))) for _ in range(2))
    v = rounded(rng.normal(size=(tokens, heads * vdim)))
    gates = rounded(rng.normal(size=(tokens, 2 * heads)) * 2.0)
    a_log = rng.uniform(np.log(0.01), np.log(4.0), size=heads).astype(np.float32)
    dt_bias = rng.uniform(-3.0, 2.0, size=heads).astype(np.float32)
    fixed = (1.0 - 2.0 ** -rng.uniform(2.0, 9.0, size=heads)).astype(np.float32)
    per_head = ops.scan_state_floats(vdim, dim)
    slots = [int(s) for s in rng.permutation(len(lengths) + 2)[:len(lengths)]]
    before = rng.normal(size=(len(lengths), heads, dim, vdim)).astype(np.float32)
    state = torch.full((len(lengths) + 2, heads * per_head + 3), 7.0, device="cuda")
    for r, slot in enumerate(slots):
        state[slot, :heads * per_head] = torch.tensor(
            packed_state(before[r], per_head).reshape(-1), dtype=torch.float32)
    o = torch.full((tokens, heads * vdim), float("nan"), device="cuda")
    scratch = torch.full((ops.delta_chunks_scratch(heads, tokens) // 4 + 1,), float("nan"),
                         device="cuda")
    starts = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    options = dict(unit_norm=True, unit_eps=1e-6, q_scale=dim ** -0.5) if unit else \
        dict(q_scale=0.5, k_scale=0.9 * dim ** -0.5)
    if unit:
        options.update(decay_in=gates[:, heads:], a_log=torch.tensor(a_log).cuda(),
                       dt_bias=torch.tensor(dt_bias).cuda())
    else:
        options.update(fixed_decay_m1=torch.tensor(fixed - 1.0).cuda())
    ops.delta_chunks(q, k, v, state, o, scratch, torch.tensor(starts).cuda(),
                     torch.tensor(slots, dtype=torch.int32).cuda(), len(lengths), tokens,
                     ops.recurrence_tiles(lengths), heads, qk_heads, dim, vdim,
                     beta_in=gates[:, :heads], **options)
    qd, kd, vd, gd = (t.double().cpu().numpy() for t in (q, k, v, gates))
    qd, kd = (x.reshape(tokens, qk_heads, dim) for x in (qd, kd))
    if unit:
        qd = qd / np.sqrt((qd * qd).sum(-1, keepdims=True) + 1e-6) * dim ** -0.5
        kd = kd / np.sqrt((kd * kd).sum(-1, keepdims=True) + 1e-6)
        log_decay = -np.exp(a_log.astype(np.float64)) * np.logaddexp(0.0, gd[:, heads:] + dt_bias)
    else:
        qd, kd = qd * 0.5, kd * np.float32(0.9 * dim ** -0.5)
        log_decay = np.broadcast_to(np.log(fixed.astype(np.float64)), (tokens, heads))
    share = heads // qk_heads
    qd, kd = np.repeat(qd, share, 1), np.repeat(kd, share, 1)
    beta = 1.0 / (1.0 + np.exp(-gd[:, :heads]))
    got_state = state.cpu().numpy()
    for r, slot in enumerate(slots):
        rows = slice(starts[r], starts[r + 1])
        want, after = plain(qd[rows], kd[rows], vd.reshape(tokens, heads, vdim)[rows], beta[rows],
                            log_decay[rows], before[r].astype(np.float64))
        # a chain of at most four float32 sums of up to 128 terms, each with a relative error of
        # 128 * 2^-24 at worst and some sqrt(128) * 2^-24 in earnest; the writes of a chunk
        # depend on one another, which multiplies it by a few
        bound = 8 * 128 ** 0.5 * 2.0 ** -24
        got = o[rows].cpu().numpy().reshape(want.shape)
        assert np.isfinite(got).all()
        assert np.linalg.norm(got - want) <= bound * np.linalg.norm(want)
        error = got_state[slot, :heads * per_head] - packed_state(after, per_head).reshape(-1)
        assert np.linalg.norm(error) <= bound * np.linalg.norm(after)
        assert (got_state[slot, heads * per_head:] == 7.0).all()
    untouched = [s for s in range(len(lengths) + 2) if s not in slots]
    assert (got_state[untouched] == 7.0).all()


def chunks_and_recurrence(q, k, v, gates, before, starts, qk_heads, a_log=None, dt_bias=None,
                          fixed=None):
    """What the chunks and what the recurrence in double make of one step of the delta rule on unit
    vectors: outputs ``[T, H, V]`` and states ``[R, H, D, V]`` of both.  ``fixed``: constant decays."""
    from helix_runtime_b200.ops import library as ops
    requests, heads, dim, vdim = before.shape
    tokens = q.shape[0]
    per_head = ops.scan_state_floats(vdim, dim)
    state = torch.tensor(np.stack([packed_state(row, per_head).reshape(-1) for row in before]),
                         dtype=torch.float32).cuda()
    o = torch.full((tokens, heads * vdim), 7.0, device="cuda")
    scratch = torch.full((ops.delta_chunks_scratch(heads, tokens) // 4 + 1,), float("nan"),
                         device="cuda")
    decays = dict(decay_in=gates[:, heads:], a_log=torch.tensor(a_log).cuda(),
                  dt_bias=torch.tensor(dt_bias).cuda()) if fixed is None else \
        dict(fixed_decay_m1=torch.tensor(fixed - 1.0, dtype=torch.float32).cuda())
    ops.delta_chunks(q, k, v, state, o, scratch, torch.tensor(starts, dtype=torch.int32).cuda(),
                     torch.arange(requests, dtype=torch.int32).cuda(), requests, tokens,
                     ops.recurrence_tiles(np.diff(starts).tolist()), heads, qk_heads, dim, vdim,
                     beta_in=gates[:, :heads], unit_norm=True, unit_eps=1e-6, **decays)
    qd, kd, vd, gd = (t.double().cpu().numpy() for t in (q, k, v, gates))
    with np.errstate(all="ignore"):
        qd, kd = (np.repeat(x / np.sqrt((x * x).sum(-1, keepdims=True) + 1e-6), heads // qk_heads, 1)
                  for x in (qd.reshape(tokens, qk_heads, dim), kd.reshape(tokens, qk_heads, dim)))
        beta = 1.0 / (1.0 + np.exp(-gd[:, :heads]))
        decay = np.broadcast_to(fixed, (tokens, heads)) if fixed is not None else \
            np.exp(-np.exp(a_log.astype(np.float64)) * np.logaddexp(0.0, gd[:, heads:] + dt_bias))
        want, after = np.zeros((tokens, heads, vdim)), before.astype(np.float64)
        for r in range(requests):
            for t in range(starts[r], starts[r + 1]):
                held = after[r] * decay[t][:, None, None]
                u = beta[t][:, None] * (vd.reshape(tokens, heads, vdim)[t] -
                                        (held * kd[t][:, :, None]).sum(1))
                after[r] = held + kd[t][:, :, None] * u[:, None]
                want[t] = (after[r] * qd[t][:, :, None]).sum(1)
    got_state = state.cpu().numpy().reshape(requests, heads, 16, vdim, -1).transpose(0, 1, 4, 2, 3)
    return o.cpu().numpy().reshape(want.shape), want, \
        got_state.reshape(requests, heads, -1, vdim)[:, :, :dim], after


def alike(got, want):
    """Not finite in the same places and alike there; elsewhere as near as the rest of this file asks."""
    assert np.array_equal(np.isnan(got), np.isnan(want))
    odd, plain_ones = np.isinf(want), np.isfinite(want)
    assert np.array_equal(got[odd], want[odd])
    error = np.linalg.norm(got[plain_ones] - want[plain_ones])
    assert error <= 8 * 128 ** 0.5 * 2.0 ** -24 * np.linalg.norm(want[plain_ones])


def inputs(rng, heads, qk_heads, dim, vdim, lengths):
    tokens = sum(lengths)
    q, k = (rounded(rng.normal(size=(tokens, qk_heads * dim))) for _ in range(2))
    v = rounded(rng.normal(size=(tokens, heads * vdim)))
    gates = rounded(rng.normal(size=(tokens, 2 * heads)))
    before = rng.normal(size=(len(lengths), heads, dim, vdim)).astype(np.float32)
    return q, k, v, gates, before, np.concatenate([[0], np.cumsum(lengths)])


@pytest.mark.parametrize("at", [37, 69])
@pytest.mark.parametrize("where", ["v inf", "v nan", "k nan", "q inf", "beta nan", "decay nan", "state inf"])
def test_what_is_not_finite_stays_behind_its_token(where, at):
    """Tokens in front of one that is not finite are what they are without it, in its chunk too; from
    it on the recurrence says what is what."""
    rng = np.random.default_rng(at)
    heads, qk_heads, dim, vdim = 4, 2, 48, 40
    q, k, v, gates, before, starts = inputs(rng, heads, qk_heads, dim, vdim, (70, 5))
    name, number = where.split()
    if name == "state":
        before[0, 1, 5, 7] = float(number)
    else:
        rows, column = {"v": (v, vdim + 3), "k": (k, 11), "q": (q, dim + 2), "beta": (gates, 1),
                        "decay": (gates, heads + 2)}[name]
        rows[at, column] = float(number)
    got, want, got_state, after = chunks_and_recurrence(
        q, k, v, gates, before, starts, qk_heads, np.linspace(-1.0, 0.5, heads).astype(np.float32),
        np.full(heads, -2.0, dtype=np.float32))
    assert not np.isfinite(want).all()
    alike(got, want)
    alike(got_state, after)


@pytest.mark.parametrize("learned", [False, True])
def test_decays_that_leave_nothing_and_negative_ones(learned):
    """Constant decays of zero and below are only factors to the recurrence; a learned one leaves
    nothing where its rate or its input is large."""
    rng = np.random.default_rng(5)
    heads, qk_heads, dim, vdim = 4, 2, 40, 24
    q, k, v, gates, before, starts = inputs(rng, heads, qk_heads, dim, vdim, (70, 5))
    if learned:
        gates[20, heads] = float("inf")
        gates[30:33, heads + 1] = 3e30
        decays = dict(a_log=np.array([0.0, 1.0, 60.0, 90.0], dtype=np.float32),
                      dt_bias=np.full(heads, -2.0, dtype=np.float32))
    else:
        decays = dict(fixed=np.array([0.0, -0.5, -1.0, 0.9]))
    got, want, got_state, after = chunks_and_recurrence(q, k, v, gates, before, starts, qk_heads, **decays)
    assert np.isfinite(want).all()
    alike(got, want)
    alike(got_state, after)


def test_constant_decays_outside_zero_to_one_take_the_scan():
    from helix_runtime_b200.parts.recurrent import LinearState
    assert LinearState.decays_suit_chunks(None) and LinearState.decays_suit_chunks([1.0, 0.5, 0.0])
    for other in (-0.25, 1.0 + 2.0 ** -23, float("nan")):
        assert not LinearState.decays_suit_chunks([0.5, other])


def test_no_further_from_64_bits_than_the_scan():
    from helix_runtime_b200.ops import library as ops
    rng = np.random.default_rng(2)
    heads, qk_heads, dim, vdim, lengths = 4, 2, 128, 128, (512, 130)
    q, k, v, gates, before, starts = inputs(rng, heads, qk_heads, dim, vdim, lengths)
    a_log = np.linspace(-2.77, 0.0, heads).astype(np.float32)
    dt_bias = np.full(heads, -2.25, dtype=np.float32)
    got, want, got_state, after = chunks_and_recurrence(q, k, v, gates, before, starts, qk_heads, a_log, dt_bias)
    per_head = ops.scan_state_floats(vdim, dim)
    state = torch.tensor(np.stack([packed_state(row, per_head).reshape(-1) for row in before]),
                         dtype=torch.float32).cuda()
    o = torch.empty((sum(lengths), heads * vdim), device="cuda")
    ops.linear_state_scan(q, k, v, state, o, torch.tensor(starts, dtype=torch.int32).cuda(),
                          torch.arange(2, dtype=torch.int32).cuda(), 2, heads, qk_heads, dim, vdim, delta=True,
                          decay_in=gates[:, heads:], beta_in=gates[:, :heads], a_log=torch.tensor(a_log).cuda(),
                          dt_bias=torch.tensor(dt_bias).cuda(), unit_norm=True, unit_eps=1e-6)
    scanned = state.cpu().numpy().reshape(2, heads, 16, vdim, -1).transpose(0, 1, 4, 2, 3).reshape(after.shape)
    scan_error = np.linalg.norm(o.cpu().numpy().reshape(want.shape) - want)
    assert np.linalg.norm(got - want) <= scan_error
    assert np.linalg.norm(got_state - after) <= np.linalg.norm(scanned - after)


@pytest.mark.parametrize("lengths", [(1, 70, 1, 1, 129), (1, 64), (3, 1, 100, 15, 16, 1), (2, 1)])
def test_portions_in_chunks_beside_the_scan_of_the_others(lengths):
    """Portions of 16 tokens and more in chunks, the other requests by the scan, to the last bit as
    if they were alone; neither touches what is the other's."""
    from helix_runtime_b200.ops import library as ops
    rng = np.random.default_rng(len(lengths))
    heads, qk_heads, dim, vdim, short = 4, 2, 48, 40, 16
    q, k, v, gates, before, starts = inputs(rng, heads, qk_heads, dim, vdim, lengths)
    tokens, requests = sum(lengths), len(lengths)
    per_head = ops.scan_state_floats(vdim, dim)
    held = torch.tensor(np.stack([packed_state(row, per_head).reshape(-1) for row in before]),
                        dtype=torch.float32).cuda()
    start = torch.tensor(starts, dtype=torch.int32).cuda()
    slots = torch.arange(requests, dtype=torch.int32).cuda()
    options = dict(decay_in=gates[:, heads:], beta_in=gates[:, :heads], unit_norm=True, unit_eps=1e-6,
                   a_log=torch.linspace(-1.0, 0.5, heads).cuda(), dt_bias=torch.full((heads,), -2.0).cuda())
    sizes = (requests, heads, qk_heads, dim, vdim)
    scanned, o_scanned = held.clone(), torch.full((tokens, heads * vdim), 7.0, device="cuda")
    ops.linear_state_scan(q, k, v, scanned, o_scanned, start, slots, *sizes, delta=True, tokens=tokens, **options)
    state, o = held.clone(), torch.full((tokens, heads * vdim), 7.0, device="cuda")
    scratch = torch.empty((ops.delta_chunks_scratch(heads, tokens),), dtype=torch.uint8, device="cuda")
    portions = [length for length in lengths if length >= short]
    ops.delta_chunks(q, k, v, state, o, scratch, start, slots, requests, tokens,
                     ops.recurrence_tiles(portions), heads, qk_heads, dim, vdim, min_query_len=short,
                     portions=len(portions), **options)
    for r, length in enumerate(lengths):
        rows = slice(starts[r], starts[r + 1])
        if length < short:
            assert (o[rows] == 7.0).all() and torch.equal(state[r], held[r])
            continue
        for got, want in ((o[rows], o_scanned[rows]), (state[r], scanned[r])):
            # both are within this of the recurrence in double (see above)
            assert (got - want).norm() <= 16 * 128 ** 0.5 * 2.0 ** -24 * want.norm()
    after_chunks, o_after_chunks = state.clone(), o.clone()
    ops.linear_state_scan(q, k, v, state, o, start, slots, *sizes, delta=True, tokens=tokens, below=short,
                          longest=max(length for length in lengths if length < short), **options)
    for r, length in enumerate(lengths):
        rows = slice(starts[r], starts[r + 1])
        same, o_same = (scanned, o_scanned) if length < short else (after_chunks, o_after_chunks)
        assert torch.equal(state[r], same[r]) and torch.equal(o[rows], o_same[rows])


@pytest.mark.parametrize("lengths,chunks_from", [
    ((1,) * 8, 0), ((31, 31), 0), ((47,), 0), ((48,), 1), ((16, 32), 1),
    ((1,) * 15 + (40,), 0),                # the scan takes all of it in the portion's time
    ((1,) * 15 + (64,), 16), ((1,) * 150 + (32,), 16), ((1, 20, 500), 16),
])
def test_a_decoding_request_does_not_take_the_chunks(lengths, chunks_from, monkeypatch):
    """What a step's requests bring decides their road: a chunk costs a decoding request as much as 64
    tokens, so portions alone go in chunks."""
    from helix_runtime_b200 import StepEntry, StepFunction
    from helix_runtime_b200.cache.manager import CacheManager
    from helix_runtime_b200.config.medolorn import DeltaMixerConfig, MedolornConfig, MedolornLayerConfig
    from helix_runtime_b200.config.registry import architecture_for
    from helix_runtime_b200.models.decoder import DecoderModel
    from helix_runtime_b200.parts import recurrent
    mixer = DeltaMixerConfig(heads=4, kv_heads=2, dim=16, vdim=16, conv=4)
    config = MedolornConfig(vocab=64, width=64, norm_eps=1e-5, canon_taps=4, max_positions=1024,
                            layers=(MedolornLayerConfig("delta", mixer, None),))
    model = DecoderModel(architecture_for(config.to_dict()).build_spec(config))
    torch.manual_seed(0)
    model.bind({request.name: torch.randn(request.shape, device="cuda").mul_(0.1).to(
        torch.float32 if request.role == "scale" else torch.bfloat16)
        for request in model.tensor_requests()}, torch.bfloat16, torch.device("cuda:0"))
    kv, state = model.cache_needs()
    cache = CacheManager(kv, state, 16, 64, len(lengths), model.max_positions, model.dtype, model.device)
    step = StepFunction(model, cache, max_tokens=sum(lengths), max_requests=len(lengths))
    for request in range(len(lengths)):
        cache.admit(request)
    routes = {}
    chunks, scan = recurrent.ops.delta_chunks, recurrent.ops.linear_state_scan

    def watched_chunks(*args, **options):
        routes["chunks"] = (options.get("min_query_len", 1), options.get("portions", args[8]))
        return chunks(*args, **options)

    def watched_scan(*args, **options):
        routes["scan"] = (options.get("below", 0), options.get("longest", 0))
        return scan(*args, **options)
    monkeypatch.setattr(recurrent.ops, "delta_chunks", watched_chunks)
    monkeypatch.setattr(recurrent.ops, "linear_state_scan", watched_scan)
    step.run([StepEntry(request, [1] * length, [length - 1]) for request, length in enumerate(lengths)])
    want = {}
    if chunks_from:
        want["chunks"] = (chunks_from, sum(length >= chunks_from for length in lengths))
    if chunks_from != 1:
        below = [length for length in lengths if length < chunks_from]
        want["scan"] = (chunks_from, max(below, default=0))
    assert routes == want


def test_refusals():
    from helix_runtime_b200.ops import library as ops
    assert ops.delta_chunks_supports(128, 8) and ops.delta_chunks_supports(8, 512)
    assert not ops.delta_chunks_supports(136, 8) and not ops.delta_chunks_supports(20, 8)
    assert not ops.delta_chunks_supports(16, 12)


@pytest.mark.parametrize("heads,qk_heads,dim,vdim", [(4, 2, 128, 128), (3, 1, 48, 136), (2, 2, 8, 8)])
def test_a_wait_that_runs_out_is_reported(heads, qk_heads, dim, vdim):
    """No polls for the rows of a portion: its status bit, NaN in every output of the portions that take chunks
    and nowhere else, the state as it was; and the next call goes on as ever."""
    from helix_runtime_b200.ops import library as ops
    torch.manual_seed(vdim)
    lengths, shortest = (70, 3, 128, 1, 65), 16
    tokens, per_head = sum(lengths), ops.scan_state_floats(vdim, dim)
    q, k = torch.randn(2, tokens, qk_heads * dim, device="cuda").bfloat16()
    v = torch.randn(tokens, heads * vdim, device="cuda").bfloat16()
    beta = torch.randn(tokens, heads, device="cuda").bfloat16()
    starts = torch.tensor(np.concatenate([[0], np.cumsum(lengths)]), dtype=torch.int32).cuda()
    slots = torch.arange(len(lengths), dtype=torch.int32, device="cuda")
    state = torch.randn(len(lengths), heads * per_head, device="cuda")
    before = state.clone()
    o = torch.full((tokens, heads * vdim), 7.0, device="cuda")
    scratch = torch.empty(ops.delta_chunks_scratch(heads, tokens) // 4 + 1, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    taken = [n for n in lengths if n >= shortest]

    def call(**options):
        ops.delta_chunks(q, k, v, state, o, scratch, starts, slots, len(lengths), tokens,
                         ops.recurrence_tiles(taken), heads, qk_heads, dim, vdim, beta_in=beta,
                         fixed_decay_m1=torch.full((heads,), -0.01, device="cuda"), unit_norm=True,
                         min_query_len=shortest, portions=len(taken), status=status, **options)

    call(polls=0)
    assert int(status.item()) == ops.FLAG_WAIT_TIMEOUT
    assert torch.equal(state, before)
    for r, n in enumerate(lengths):
        rows = o[starts[r]:starts[r + 1]]
        assert rows.isnan().all() if n >= shortest else (rows == 7.0).all()
    status.zero_()
    call()
    assert int(status.item()) == 0 and o.isfinite().all() and state.isfinite().all()
    changed = [not torch.equal(state[r], before[r]) for r in range(len(lengths))]
    assert changed == [n >= shortest for n in lengths]
