"""Matrix memories over prompts in chunks on the tensor cores, against the recurrence in 64 bits and against the row-by-row scan.

Inputs to both are the same bfloat16 (or float32) numbers, products keep float32's 24 bits and sums are float32, so a result may
be off by the rounding of sums of a few hundred terms: 2e-6 of the largest output is about ten roundings of 2^-24.
"""
import pytest
import torch

from quicknn_b200.kernels import ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
TOL = 2e-6


def recurrence(q, k, v, decay, w, scale, state, row0, lens, slots, ones):
    """Row by row in 64 bits: q, k [T, H, D], v [T, H, V], decay [T, H, D or 1], w [T, H] -> out [T, H, V (+1)], states."""
    T, H, D = q.shape
    v = torch.cat([v, torch.ones_like(v[..., :1])], -1) if ones else v
    out = torch.zeros((T, H, v.shape[-1]), dtype=torch.float64, device=DEV)
    state = state.double().clone()
    for r0, n, s in zip(row0, lens, slots):
        if s < 0:
            continue
        S = state[s]
        for t in range(r0, r0 + n):
            S = decay[t][..., None] * S + (w[t][:, None] * k[t])[..., None] * v[t][:, None, :]
            out[t] = ((q[t] * scale)[:, None, :] @ S)[:, 0]
        state[s] = S
    return out, state


def inputs(lens, H, D, V, seed, dtype=torch.bfloat16):
    torch.manual_seed(seed)
    T = sum(lens)
    proj = torch.randn((T, H * (2 * D + V) + 8), device=DEV).to(dtype)
    row0 = [sum(lens[:i]) for i in range(len(lens))]
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    q, k, v = (t.double() for t in proj[:, :H * (2 * D + V)].split([H * D, H * D, H * V], 1))
    return proj, row0, i32(row0), i32(lens), q.reshape(T, H, D), k.reshape(T, H, D), v.reshape(T, H, V)


def off(got, want):
    """(largest difference over the largest value, 2-norm of the difference over that of the value)"""
    d = got.double() - want
    return (d.abs().max() / want.abs().max()).item(), (d.norm() / want.norm()).item()


def everything_in_chunks(monkeypatch):
    monkeypatch.setattr(ops, "MEMORY_CHUNKS_FREE", 1 << 30)
    for name in ("MEMORY_CHUNKS_FROM", "MEMORY_CHUNKS_FROM_WIDE"):
        monkeypatch.setattr(ops, name, 1)


# lengths about the edges of a chunk (64) and a sub-chunk (16), the longest first, last and among others; slot -1: no sequence
LENGTHS = [([64], [0]), ([1, 65, 16], [2, 0, 3]), ([79, 128, 17], [1, -1, 0]), ([321], [3]), ([15, 200, 63, 64], [0, 1, 2, 3])]


@pytest.mark.parametrize("lens,slots", LENGTHS)
@pytest.mark.parametrize("D,V", [(64, 8), (64, 128), (128, 24), (128, 256)])
@pytest.mark.parametrize("kind", ["channels", "complement", "constant", "gates", "float_keys"])
@pytest.mark.parametrize("at_once", [1, 2, 3, 1000])             # chunks of a round, of one sequence or several; the last round may have fewer
def test_chunks_against_64_bits(lens, slots, D, V, kind, at_once, monkeypatch):
    H, T = 3, sum(lens)
    proj, row0, d_row0, d_lens, q, k, v = inputs(lens, H, D, V, 5 + D + V + T)
    monkeypatch.setattr(ops, "MEMORY_CHUNKS_SCRATCH", 4 * H * D * V * at_once)
    everything_in_chunks(monkeypatch)
    ones = kind == "gates"
    state = torch.randn((4, H, D, V + ones), device=DEV)
    d_slots = torch.tensor(slots, dtype=torch.int32, device=DEV)
    w = torch.ones((T, H), device=DEV)
    if kind in ("channels", "complement"):
        # from no decay at all to one that leaves nothing, channel by channel
        decay = torch.rand((T, H, D), device=DEV) ** (torch.arange(D, device=DEV) % 5).float()
        decay[:, :, 1::11] = 0.0
        decay[T // 2, :, ::7] = 1e-38
        key = 1.0 - decay.double() if kind == "complement" else k
        want, end = recurrence(q, key, v, decay.double(), w.double(), D ** -0.5, state, row0, lens, slots, False)
        run = lambda st, longest: ops.gla_scan(proj, 0, H * D, 2 * H * D, decay.reshape(T, H * D), D ** -0.5, d_row0, d_lens,  # noqa: E731
                                               d_slots, st, len(lens), H, D, V, longest=longest, key_from_decay=kind == "complement")
    else:
        gates = torch.rand((T, 2 * H), device=DEV)
        decay = gates[:, :H]
        rows, values, ld, flat = proj, None, 2 * H, gates
        if kind == "constant":
            flat = torch.tensor([1.0, 0.97, 0.01], device=DEV)
            ld, decay = 0, flat.expand(T, H)
        if kind == "gates":
            w = gates[:, H:]
        if kind == "float_keys":
            rows = torch.randn((T, 2 * H * D), device=DEV)
            q, k = (x.double().reshape(T, H, D) for x in rows.split(H * D, 1))
            values = proj
        want, end = recurrence(q, k, v, decay.double()[..., None], w.double(), D ** -0.5, state, row0, lens, slots, ones)
        wide = torch.cat([rows, proj[:, 2 * H * D:2 * H * D + H * V].float()], 1) if values is not None else proj

        def run(st, longest):
            own = values is not None and longest > 0
            return ops.memory_scan(rows if own else wide, 0, H * D, 2 * H * D, flat, ld, gates if ones else None, H, D ** -0.5, ones,
                                   d_row0, d_lens, d_slots, st, len(lens), H, D, V, longest=longest, values=values if own else None)
    results = []
    for longest in (max(lens), 0):                               # in chunks; row by row
        st = state.clone() if kind in ("channels", "complement") else state.reshape(4, -1).clone()
        out = run(st, longest)
        results.append(off(out.reshape(want.shape), want) + off(st.reshape(end.shape), end))
        assert all((st.reshape(end.shape)[s] == state[s]).all() for s in range(4) if s not in slots)
    assert max(results[0]) < TOL, results
    # no less precise than the walk: but for the one rounding more (2^-24) of queries and keys times their decays
    assert results[0][1] <= results[1][1] + 2 ** -24 and results[0][3] <= results[1][3] + 2 ** -24, results


@pytest.mark.parametrize("place", ["value", "key", "query", "decay", "state"])
@pytest.mark.parametrize("bad", [float("inf"), float("-inf"), float("nan")])
@pytest.mark.parametrize("kind", ["channels", "gates", "float_keys"])
def test_numbers_that_are_not_finite_stay_where_they_belong(kind, bad, place, monkeypatch):
    """Inf or NaN in one number: the results that are not finite are those of the walk, and all others are what they are without it."""
    everything_in_chunks(monkeypatch)
    H, D, V, lens, slots = 2, 64, 40, [150, 70], [1, 0]
    T, ones = sum(lens), kind == "gates"
    proj, row0, d_row0, d_lens, q, k, v = inputs(lens, H, D, V, 11)
    rows = torch.cat([torch.randn((T, 2 * H * D), device=DEV), proj[:, 2 * H * D:2 * H * D + H * V].float()], 1) if kind == "float_keys" else proj
    if kind == "float_keys":
        q, k = (x.double().reshape(T, H, D) for x in rows[:, :2 * H * D].split(H * D, 1))
    gates = 0.5 + 0.5 * torch.rand((T, H * D if kind == "channels" else 2 * H), device=DEV)
    start = torch.randn((2, H, D, V + ones), device=DEV)
    d_slots = torch.tensor(slots, dtype=torch.int32, device=DEV)
    dec = gates.double().reshape(T, H, D) if kind == "channels" else gates[:, :H, None].double()
    w = gates[:, H:].double() if ones else torch.ones((T, H), device=DEV).double()
    clean, _ = recurrence(q, k, v, dec, w, D ** -0.5, start, row0, lens, slots, ones)
    for at in (0, 5, 15, 37, 63, 64, 149, 150, 215):             # rows of the first and of the second sequence
        p, r, g, st = proj.clone(), rows.clone(), gates.clone(), start.clone()
        if place == "value":
            p[at, 2 * H * D + V + 3] = bad                       # head 1, column 3
            r[at, 2 * H * D + V + 3] = bad
        elif place in ("key", "query"):
            c = (H * D if place == "key" else 0) + D + 7         # head 1, channel 7
            p[at, c] = bad
            r[at, c] = bad
        elif place == "decay":
            g[at, D + 7 if kind == "channels" else 1] = bad
        else:
            st[at % 2, 1, 7, 3] = bad
        got = []
        for longest in (max(lens), 0):
            s = st.clone() if kind == "channels" else st.reshape(2, -1).clone()
            if kind == "channels":
                out = ops.gla_scan(p, 0, H * D, 2 * H * D, g, D ** -0.5, d_row0, d_lens, d_slots, s, 2, H, D, V, longest=longest)
            else:
                own = kind == "float_keys" and longest > 0
                src = r if kind == "float_keys" else p
                out = ops.memory_scan(src, 0, H * D, 2 * H * D, g, 2 * H, g if ones else None, H, D ** -0.5, ones, d_row0, d_lens, d_slots, s, 2,
                                      H, D, V, longest=longest, values=p if own else None)
            got.append((out.reshape(clean.shape), s.reshape(start.shape)))
        (out, s), (walked, s_walked) = got
        fine = walked.isfinite()
        assert torch.equal(out.isfinite(), fine) and torch.equal(s.isfinite(), s_walked.isfinite()), at
        assert not fine.all() and fine.any()
        assert ((out.double() - clean)[fine].abs().max() / clean.abs().max()).item() < TOL, at


@pytest.mark.parametrize("lens,slots", [([1, 300, 47, 48, 1], [0, 1, 2, 3, 4]), ([1] * 40 + [241] + [2] * 9 + [64, 130], [-1] + list(range(1, 52)))])
@pytest.mark.parametrize("D,V", [(64, 24), (128, 64)])
@pytest.mark.parametrize("kind", ["channels", "gates", "float_keys"])
def test_short_sequences_beside_a_prompt_walk(lens, slots, D, V, kind, monkeypatch):
    """A step of unequal sequences: the long ones run in chunks, one among many others included; those of a few rows walk, and give the
    walk's results bit for bit."""
    monkeypatch.setattr(ops, "MEMORY_CHUNKS_FREE", 0)            # as if the heads were many
    H, T, ones = 2, sum(lens), kind == "gates"
    proj, row0, d_row0, d_lens, q, k, v = inputs(lens, H, D, V, 3)
    rows = proj
    if kind == "float_keys":
        rows = torch.cat([torch.randn((T, 2 * H * D), device=DEV), proj[:, 2 * H * D:2 * H * D + H * V].float()], 1)
        q, k = (x.double().reshape(T, H, D) for x in rows[:, :2 * H * D].split(H * D, 1))
    gates = 0.5 + 0.5 * torch.rand((T, H * D if kind == "channels" else 2 * H), device=DEV)
    start = torch.randn((len(lens), H, D, V + ones), device=DEV)
    d_slots = torch.tensor(slots, dtype=torch.int32, device=DEV)
    dec = gates.double().reshape(T, H, D) if kind == "channels" else gates[:, :H, None].double()
    w = gates[:, H:].double() if ones else torch.ones((T, H), device=DEV).double()
    want, end = recurrence(q, k, v, dec, w, D ** -0.5, start, row0, lens, slots, ones)
    got = []
    for longest, shortest in ((max(lens), min(lens)), (max(lens), 0), (0, 0)):
        s = start.clone() if kind == "channels" else start.reshape(len(lens), -1).clone()
        if kind == "channels":
            out = ops.gla_scan(proj, 0, H * D, 2 * H * D, gates, D ** -0.5, d_row0, d_lens, d_slots, s, len(lens), H, D, V, longest=longest,
                               shortest=shortest)
        else:
            out = ops.memory_scan(rows, 0, H * D, 2 * H * D, gates, 2 * H, gates if ones else None, H, D ** -0.5, ones, d_row0, d_lens,
                                  d_slots, s, len(lens), H, D, V, longest=longest, shortest=shortest,
                                  values=proj if kind == "float_keys" and longest > 0 else None)
        got.append((out.reshape(want.shape), s.reshape(start.shape)))
        assert max(off(got[-1][0], want) + off(got[-1][1], end)) < TOL
    for out, s in got[:2]:
        for r0, n, slot in zip(row0, lens, slots):
            same = torch.equal(out[r0:r0 + n], got[2][0][r0:r0 + n])
            assert same if n < ops.MEMORY_CHUNKS_BESIDE or slot < 0 else not same, (n, slot)
            if n < ops.MEMORY_CHUNKS_BESIDE and slot >= 0:
                assert torch.equal(s[slot], got[2][1][slot])


def test_scratch_has_a_limit():
    """A prompt beside many sequences: the scratch is bounded whatever their number."""
    lens, H, D, V = [1] * 71 + [200], 9, 128, 256
    proj, row0, d_row0, d_lens, *_ = inputs(lens, H, D, V, 2)
    gates, state = torch.rand((sum(lens), 2 * H), device=DEV), torch.zeros((72, H * D * V), device=DEV)
    d_slots = torch.arange(72, dtype=torch.int32, device=DEV)
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    out = ops.memory_scan(proj, 0, H * D, 2 * H * D, gates, 2 * H, None, 0, 1.0, False, d_row0, d_lens, d_slots, state, 72, H, D, V, longest=200)
    # 271 rows are at most nine chunks, if five sequences of 48 rows and more have a short last one; a chunk per sequence were 72
    assert torch.cuda.max_memory_allocated() - before <= 4 * out.numel() + 9 * 4 * H * D * V + (1 << 20)


def test_what_is_refused_or_walks():
    """Other sizes, float32 values and short steps keep the row-by-row scan; a step that walks takes no values of its own."""
    bf = torch.bfloat16
    assert ops.memory_chunks_fit(bf, 64, 128, 96, 8, 16) and ops.memory_chunks_fit(bf, 128, 128, 160, per_channel=True)
    for case in ((torch.float32, 64, 128, 96, 8), (bf, 96, 128, 96, 8), (bf, 64, 257, 96, 8), (bf, 64, 264, 96, 8), (bf, 64, 128, 95, 8),
                 (bf, 64, 128, 96, 4)):
        assert not ops.memory_chunks_fit(*case)
    proj, _, d_row0, d_lens, *_ = inputs([20], 2, 64, 16, 1)
    with pytest.raises(ValueError):
        ops.memory_scan(proj, 0, 128, 256, torch.ones(2, device=DEV), 0, None, 0, 1.0, False, d_row0, d_lens,
                        torch.zeros(1, dtype=torch.int32, device=DEV), torch.zeros((1, 2 * 64 * 16), device=DEV), 1, 2, 64, 16, longest=20,
                        values=proj)
