"""GPU: the forward pass over compact records at the sizes where its kernels can go wrong - around the 32-token chunk, its
16-token halves and the rings of the copies; batches on either side of the lines between the forms of the recurrence (a chain
split over four or two CTAs, one CTA per chain, two time slices, the persistent form, runs); empty sequences; every state form."""
import pytest
import torch

import flashkda_b200 as F
import oracle
from flashkda_b200.workloads import Workload, make_inputs
from helpers import OUT_MAX_ABS, STATE_REL, max_abs, rel_fro, to_cuda

pytestmark = pytest.mark.gpu

CASES = {
    "chunk_edges_split4": Workload("c", H=3, seq_lens=[1, 15, 16, 17, 31, 32, 33, 63, 64, 65, 97], state_in="fp32", state_out="fp32"),
    "ring_lengths_split4": Workload("c", H=2, B=3, T=32 * 9 + 5, state_in="bf16", state_out="bf16"),
    "split2": Workload("c", H=25, B=2, T=33 + 64, state_out="fp32"),
    "one_cta": Workload("c", H=40, B=3, T=32 * 6 + 1, state_in="fp32", state_out="fp32"),
    "one_cta_no_state": Workload("c", H=100, B=1, T=48),
    "persistent_two_rounds": Workload("c", H=50, B=6, T=70, state_in="bf16", state_out="bf16"),
    "persistent_packed_with_empty": Workload("c", H=16, seq_lens=[0, 5, 33, 0, 64, 1, 31, 32, 100, 0, 2, 47], state_in="fp32", state_out="fp32"),
    "two_slices": Workload("c", H=30, B=3, T=32 * 140 + 7, state_in="fp32", state_out="fp32"),
    "two_slices_no_state": Workload("c", H=80, B=1, T=32 * 150),
    "runs": Workload("c", H=2, B=1, T=32 * 700 + 9, state_in="fp32", state_out="fp32", lower_bound=-1.0),
}


@pytest.mark.parametrize("name", list(CASES))
def test_compact_path_matches_the_recurrence(name):
    w = CASES[name]
    x = make_inputs(w)
    xc = to_cuda(x)
    out = torch.full_like(xc["v"], float("nan"))
    fin = None if xc["final_state"] is None else torch.full_like(xc["final_state"], float("nan"))
    B, T = x["q"].shape[:2]
    ws = torch.empty(F.get_workspace_size(B * T, w.H, w.N), dtype=torch.uint8, device="cuda")
    args = (xc["q"], xc["k"], xc["v"], xc["g"], xc["beta"], x["scale"], out, xc["A_log"], xc["dt_bias"], x["lower_bound"])
    kw = dict(initial_state=xc["initial_state"], final_state=fin, cu_seqlens=xc["cu_seqlens"])
    F.fwd(*args, workspace=ws, **kw)
    assert F.read_status(ws) == 0
    o64, s64 = oracle.recurrence_f64(x["q"], x["k"], x["v"], x["g"], x["beta"], x["scale"], x["A_log"], x["dt_bias"], x["lower_bound"],
                                     initial_state=x["initial_state"], cu_seqlens=x["cu_seqlens"])
    assert max_abs(out.cpu(), o64) <= OUT_MAX_ABS and rel_fro(out.cpu(), o64) <= 1e-2
    if fin is not None:
        assert rel_fro(fin.cpu(), s64) <= STATE_REL
    # and again through the plain call, and stage by stage: same bits
    first, first_fin = out.clone(), None if fin is None else fin.clone()
    out.fill_(float("nan"))
    F.operands(*args, cu_seqlens=xc["cu_seqlens"], workspace=ws)
    F.recurrence(*args, workspace=ws, **kw)
    assert F.read_status(ws) == 0
    assert torch.equal(out.view(torch.int16), first.view(torch.int16)) and (fin is None or torch.equal(fin, first_fin))
    F.fwd(*args, **kw)
    assert torch.equal(out.view(torch.int16), first.view(torch.int16)) and (fin is None or torch.equal(fin, first_fin))


@pytest.mark.parametrize("case", ["fixed_many_items", "packed_many_sequences", "tails"])
def test_operands_kernel_gives_the_bits_of_its_one_item_per_cta_form(case):
    """A CTA of the token-parallel kernel reuses tile slots, operands, accumulators, staging and barrier phases over many items;
    with one item per CTA nothing is reused.  A stale tile, a buffer overwritten too early or a lost phase would show in the
    results of the call: up to 74 items per CTA, ragged sequences, repeated calls."""
    if case == "fixed_many_items":
        w = Workload("o1", H=32, B=4, T=5400, state_out="fp32", seed=21)
    elif case == "packed_many_sequences":
        import random
        rnd = random.Random(5)
        w = Workload("o2", H=8, seq_lens=[rnd.choice([0, 1, 7, 31, 32, 33, 63, 64, 65, 100, 257, 1000]) for _ in range(300)], state_out="fp32", seed=22)
    else:
        w = Workload("o3", H=5, B=7, T=32 * 40 + 3, state_in="bf16", state_out="bf16", seed=23)
    x = make_inputs(w, device="cuda")

    def call(flags):
        out, fin = torch.full_like(x["v"], float("nan")), torch.full_like(x["final_state"], float("nan"))
        ws = torch.empty(F.get_workspace_size(x["q"].shape[0] * x["q"].shape[1], w.H, w.N), dtype=torch.uint8, device="cuda")
        F.fwd(x["q"], x["k"], x["v"], x["g"], x["beta"], x["scale"], out, x["A_log"], x["dt_bias"], x["lower_bound"],
              initial_state=x["initial_state"], final_state=fin, cu_seqlens=x["cu_seqlens"], workspace=ws, flags=flags)
        assert F.read_status(ws) == 0
        return out, fin

    out, fin = call(F.FLAG_OPERANDS_PER_ITEM)
    assert not torch.isnan(out.float()).any() and not torch.isnan(fin.float()).any()
    for _ in range(3):
        o, f = call(0)
        assert torch.equal(o.view(torch.int16), out.view(torch.int16)) and torch.equal(f, fin)


def test_a_wait_in_operands_kernel_gives_up_and_the_context_stays_usable():
    """Every CTA loads the tiles of its first item only and the waits are given three milliseconds.  With 600 items some CTAs
    have a second one whose tiles never come: the call must return with status 2 and its tensor memory released, which the
    ordinary call behind it needs.  With an item per CTA nobody meets the missing load.  Nothing faults, and what a CTA has in
    flight when it gives up (its first item's products and stores) has ended before it leaves."""
    for T, status in ((32 * 600, 2), (32 * 200, 0)):
        w = Workload("g", H=1, T=T, state_out="fp32", seed=6)
        x = make_inputs(w, device="cuda")
        args = (x["q"], x["k"], x["v"], x["g"], x["beta"], x["scale"], x["out"], x["A_log"], x["dt_bias"], x["lower_bound"])
        ws = torch.empty(F.get_workspace_size(T, 1, 1), dtype=torch.uint8, device="cuda")
        F.fwd(*args, final_state=x["final_state"], workspace=ws)
        assert F.read_status(ws) == 0
        out, fin = x["out"].clone(), x["final_state"].clone()
        F.operands(*args, workspace=ws, wait_limit_us=3000)
        if status:
            with pytest.raises(RuntimeError, match="bounded wait"):
                F.read_status(ws)
        else:
            assert F.read_status(ws) == 0
        F.fwd(*args, final_state=x["final_state"], workspace=ws)
        assert F.read_status(ws) == 0
        assert torch.equal(x["out"].view(torch.int16), out.view(torch.int16)) and torch.equal(x["final_state"], fin)


def test_benchmark_counts_the_kernels_that_a_call_launches():
    """bench.py's count, from a graph captured around a call: one kernel for a step of a few tokens, two for a prefill, four with
    runs (two passes and the chaining of their maps), three in a packed batch plus the one for its decode tokens."""
    from bench import kernels_per_call, make_caller
    for w, n in ((Workload("k", H=4, B=3, T=1, state_out="fp32"), 1), (Workload("k", H=4, B=3, T=300, state_out="fp32"), 2),
                 (Workload("k", H=2, T=32 * 700, state_out="fp32"), 4), (Workload("k", H=4, seq_lens=[300, 1, 70], state_out="fp32"), 4)):
        x = make_inputs(w, device="cuda")
        ws = torch.empty(F.get_workspace_size(x["q"].shape[0] * x["q"].shape[1], w.H, w.N), dtype=torch.uint8, device="cuda")
        call = make_caller(F, x, ws, 0)
        call()
        assert kernels_per_call(call) == n, w


@pytest.mark.parametrize("w", [Workload("d", H=4, B=3, T=1, state_in="fp32", state_out="fp32"), Workload("p", H=3, B=2, T=300, state_out="fp32"),
                               Workload("s", H=80, T=32 * 128, state_out="fp32"), Workload("r", H=2, T=32 * 700, state_out="fp32"),
                               Workload("v", H=12, seq_lens=[1, 40, 4, 300, 1, 33], state_in="bf16", state_out="bf16")],
                         ids=["decode", "prefill", "two_slices", "runs", "packed_with_decode"])
def test_captured_call_replays_on_new_inputs(w):
    """The plain call in a CUDA graph (scratch memory from the graph's pool, kernels that start beside their predecessors):
    replays on other inputs in the same buffers give the bits of ordinary calls."""
    x = make_inputs(w, device="cuda")
    args = (x["q"], x["k"], x["v"], x["g"], x["beta"], x["scale"], x["out"], x["A_log"], x["dt_bias"], x["lower_bound"])
    kw = dict(initial_state=x["initial_state"], final_state=x["final_state"], cu_seqlens=x["cu_seqlens"])
    F.fwd(*args, **kw)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        F.fwd(*args, **kw)
    for seed in (1, 2):
        gen = torch.Generator(device="cuda").manual_seed(seed)
        for name in ("q", "k", "v", "g", "beta"):
            x[name].copy_(torch.randn(x[name].shape, generator=gen, device="cuda"))
        F.fwd(*args, **kw)
        out, fin = x["out"].clone(), x["final_state"].clone()
        x["out"].fill_(float("nan"))
        x["final_state"].fill_(float("nan"))
        graph.replay()
        assert torch.equal(x["out"].view(torch.int16), out.view(torch.int16)) and torch.equal(x["final_state"], fin)


GIVEUP = {
    "split4": (Workload("g", H=3, B=2, T=200, state_in="fp32", state_out="fp32", seed=1), 2),
    "split2": (Workload("g", H=25, B=2, T=200, state_out="fp32", seed=2), 3),
    "one_cta": (Workload("g", H=50, B=2, T=300, state_in="bf16", state_out="bf16", seed=3), 4),
    "persistent": (Workload("g", H=50, B=6, T=200, state_out="fp32", seed=4), 9),
    "packed_with_decode": (Workload("g", H=40, seq_lens=[1, 200, 40, 3, 300, 64], state_in="fp32", state_out="fp32", seed=5), 1),
    "slices": (Workload("g", H=80, T=32 * 128, state_out="fp32", seed=6), 7),
    "runs": (Workload("g", H=2, T=32 * 700, state_out="fp32", lower_bound=-1.0, seed=7), 6),
    "chaining": (Workload("g", H=2, T=32 * 700, state_out="fp32", lower_bound=-1.0, seed=7), -4),
}


@pytest.mark.parametrize("form", list(GIVEUP))
def test_a_wait_in_the_recurrence_gives_up_and_the_context_stays_usable(form):
    """Each form of the recurrence with copies that stop in the middle of a walk and waits of three milliseconds: the call must
    return with status 2, and the ordinary call behind it, which needs all of the tensor memory, gives the bits of the one
    before.  Nothing faults and nothing is in flight when a wait runs out."""
    w, stop = GIVEUP[form]
    x = make_inputs(w, device="cuda")
    args = (x["q"], x["k"], x["v"], x["g"], x["beta"], x["scale"], x["out"], x["A_log"], x["dt_bias"], x["lower_bound"])
    kw = dict(initial_state=x["initial_state"], final_state=x["final_state"], cu_seqlens=x["cu_seqlens"])
    ws = torch.empty(F.get_workspace_size(x["q"].shape[0] * x["q"].shape[1], w.H, w.N), dtype=torch.uint8, device="cuda")
    F.fwd(*args, workspace=ws, **kw)
    assert F.read_status(ws) == 0
    out, fin = x["out"].clone(), x["final_state"].clone()
    F.recurrence_giveup(*args, workspace=ws, stop_copies_after=stop, **kw)
    with pytest.raises(RuntimeError, match="bounded wait"):
        F.read_status(ws)
    F.recurrence_giveup(*args, workspace=ws, stop_copies_after=1000000 if stop > 0 else -1000000, wait_limit_us=1000000, **kw)     # (held back by nothing)
    assert F.read_status(ws) == 0
    F.fwd(*args, workspace=ws, **kw)
    assert F.read_status(ws) == 0
    assert torch.equal(x["out"].view(torch.int16), out.view(torch.int16)) and torch.equal(x["final_state"], fin)


@pytest.mark.parametrize("H,T,packed", [(24, 8192, False), (8, 8192, False), (4, 20000, False), (2, 12000, True)])
def test_the_call_walks_the_runs_that_the_planner_reports(H, T, packed):
    """The slots behind the records show how many runs a call has made: the state at the start of every run but the first is in
    its slot, and nothing is written behind the slots of the reported number of runs.  (Packed: two sequences of T tokens,
    planned for a third more.)"""
    N = 2 if packed else 1
    w = Workload("plan", H=H, T=T, seq_lens=[T, T] if packed else None, state_out="fp32", seed=H)
    x = make_inputs(w, device="cuda")
    runs, _ = F.plan_segments(N * H, ((T * 4 // 3 if packed else T) + 31) // 32)
    off, rec, per_head = F.workspace_layout(N * T, H, N, packed, T)
    slots, slot = off + rec * per_head * H, 3 * 128 * 136 * 4
    size = max(F.get_workspace_size(N * T, H, N), slots) + 2 * N * H * slot
    ws = torch.full((size,), 0x5A, dtype=torch.uint8, device="cuda")
    F.fwd(x["q"], x["k"], x["v"], x["g"], x["beta"], x["scale"], x["out"], x["A_log"], x["dt_bias"], x["lower_bound"],
          final_state=x["final_state"], cu_seqlens=x["cu_seqlens"], workspace=ws)
    assert F.read_status(ws) == 0
    used = runs if runs > 1 else 0
    assert bool((ws[slots + used * N * H * slot:] == 0x5A).all()), "more runs than reported"
    if used:
        states = ws[slots:slots + used * N * H * slot].view(N * H, used, 3, 128 * 136 * 4)[:, 1:, 2, :128 * 128 * 4]
        assert bool((states != 0x5A).any(-1).all()), "fewer runs than reported"


@pytest.mark.parametrize("state", ["bf16", "fp32"])
@pytest.mark.parametrize("H,T,lens", [(2, 32 * 700, None), (8, 8192, None), (2, 0, [32 * 200 + 9, 0, 32 * 180, 32 * 3 + 1]), (3, 0, [9000, 40])],
                         ids=["two_heads", "eight_heads", "packed", "packed_empty_last_runs"])
def test_states_may_be_updated_in_place_by_calls_that_are_cut_into_runs(H, T, lens, state):
    """`initial_state is final_state`, as a server keeps them: the bits of a call with separate tensors.  The last run, which in the packed
    batches is empty for the shorter sequence and stores at once, works beside run 0; so run 0 starts from the copy that the first
    pass has left in its slot."""
    w = Workload("in place", H=H, T=T, seq_lens=lens, state_in=state, state_out=state, state_std=0.5, seed=H)
    x = make_inputs(w, device="cuda")
    args = (x["q"], x["k"], x["v"], x["g"], x["beta"], x["scale"], x["out"], x["A_log"], x["dt_bias"], x["lower_bound"])
    tokens, chains = x["q"].shape[1], w.N * H
    runs = F.plan_segments(chains, (tokens // w.N + 31) // 32)[0]
    if lens:
        runs = min(runs, F.plan_segments(chains, (tokens * 4 // (w.N * 3) + 31) // 32)[0])
    assert runs > 1
    off, rec, per_head = F.workspace_layout(tokens, H, w.N, lens is not None, T)
    slots, floats = off + rec * per_head * H, 128 * 136
    ws = torch.full((max(F.get_workspace_size(tokens, H, w.N), slots + chains * runs * 3 * floats * 4),), 0xFF, dtype=torch.uint8, device="cuda")
    before = x["initial_state"].clone()
    F.fwd(*args, initial_state=x["initial_state"], final_state=x["final_state"], cu_seqlens=x["cu_seqlens"], workspace=ws)
    assert F.read_status(ws) == 0
    assert torch.equal(x["initial_state"], before)
    taken = ws[slots:slots + chains * runs * 3 * floats * 4].view(torch.float32).view(w.N, H, runs, 3, floats)[:, :, 0, 2, :128 * 128]
    taken = taken.reshape(before.shape)
    for n in range(w.N):
        if lens is None or lens[n] > 4:          # (the others are the per-token kernel's)
            assert torch.equal(taken[n], before[n].float()), n
    out, fin = x["out"].clone(), x["final_state"].clone()
    for _ in range(20):
        both = before.clone()
        F.fwd(*args, initial_state=both, final_state=both, cu_seqlens=x["cu_seqlens"], workspace=ws)
        assert torch.equal(x["out"].view(torch.int16), out.view(torch.int16)) and torch.equal(both, fin)


@pytest.mark.parametrize("state", [None, "bf16", "fp32"])
@pytest.mark.parametrize("B,T", [(1, 1), (3, 4), (2, 5), (5, 15), (5, 16), (3, 17), (2, 31), (2, 32), (400, 3)])
def test_short_sequences_match_the_recurrence(B, T, state):
    """The per-token kernel (quarters of a chain, whole chains) and the 16-token tile kernel (one block, two blocks) on either
    side of the lines between them."""
    w = Workload("s", H=2, B=B, T=T, state_in=state, state_out=state or "fp32", state_std=0.5, seed=B * 100 + T, lower_bound=-2.0)
    x = make_inputs(w)
    xc = to_cuda(x)
    out = torch.full_like(xc["v"], float("nan"))
    fin = torch.full_like(xc["final_state"], float("nan"))
    F.fwd(xc["q"], xc["k"], xc["v"], xc["g"], xc["beta"], x["scale"], out, xc["A_log"], xc["dt_bias"], x["lower_bound"],
          initial_state=xc["initial_state"], final_state=fin)
    o64, s64 = oracle.recurrence_f64(x["q"], x["k"], x["v"], x["g"], x["beta"], x["scale"], x["A_log"], x["dt_bias"], x["lower_bound"],
                                     initial_state=x["initial_state"])
    assert max_abs(out.cpu(), o64) <= OUT_MAX_ABS and rel_fro(out.cpu(), o64) <= 1e-2
    assert rel_fro(fin.cpu(), s64) <= STATE_REL


@pytest.mark.parametrize("state", [None, "bf16", "fp32"])
@pytest.mark.parametrize("B,T", [(3, 5), (3, 6), (5, 7), (3, 8), (3, 9), (300, 8)])
def test_eight_token_tiles_match_the_recurrence(B, T, state):
    """The eight-token form of the tile kernel, around its edges, with and without a final state."""
    w = Workload("e", H=2, B=B, T=T, state_in=state, state_out=state or "fp32", state_std=0.5, seed=B * 100 + T, lower_bound=-2.0)
    x = make_inputs(w)
    xc = to_cuda(x)
    out, fin = torch.full_like(xc["v"], float("nan")), torch.full_like(xc["final_state"], float("nan"))
    for final in (fin, None):
        F.fwd(xc["q"], xc["k"], xc["v"], xc["g"], xc["beta"], x["scale"], out, xc["A_log"], xc["dt_bias"], x["lower_bound"],
              initial_state=xc["initial_state"], final_state=final)
        o64, s64 = oracle.recurrence_f64(x["q"], x["k"], x["v"], x["g"], x["beta"], x["scale"], x["A_log"], x["dt_bias"], x["lower_bound"],
                                         initial_state=x["initial_state"])
        assert max_abs(out.cpu(), o64) <= OUT_MAX_ABS and rel_fro(out.cpu(), o64) <= 1e-2
    assert rel_fro(fin.cpu(), s64) <= STATE_REL


def test_decode_tokens_among_prompts():
    """A packed batch that mixes sequences of a few tokens, which the per-token kernel takes, with prompts."""
    lens = [1] * 7 + [40, 4, 5, 0, 300, 1, 3, 33]
    w = Workload("m", H=12, seq_lens=lens, state_in="bf16", state_out="bf16", state_std=0.5, seed=77)
    x = make_inputs(w)
    xc = to_cuda(x)
    out, fin = torch.full_like(xc["v"], float("nan")), torch.full_like(xc["final_state"], float("nan"))
    F.fwd(xc["q"], xc["k"], xc["v"], xc["g"], xc["beta"], x["scale"], out, xc["A_log"], xc["dt_bias"], x["lower_bound"],
          initial_state=xc["initial_state"], final_state=fin, cu_seqlens=xc["cu_seqlens"])
    o64, s64 = oracle.recurrence_f64(x["q"], x["k"], x["v"], x["g"], x["beta"], x["scale"], x["A_log"], x["dt_bias"], x["lower_bound"],
                                     initial_state=x["initial_state"], cu_seqlens=x["cu_seqlens"])
    assert max_abs(out.cpu(), o64) <= OUT_MAX_ABS
    assert rel_fro(fin.cpu(), s64) <= STATE_REL
    assert torch.equal(fin[lens.index(0)].cpu(), x["initial_state"][lens.index(0)])


@pytest.mark.parametrize("lens", [[33, 40, 1, 20, 97, 31], [47, 5, 63, 70, 16, 100, 17]])
def test_rows_past_a_sequence_end_do_not_matter(lens):
    """The last tile of a sequence holds the first rows of the next one: whatever these are, not-a-number included, the results of
    the sequence are the same bits.  (Every other sequence is spoilt in turn.)"""
    w = Workload("n", H=6, seq_lens=lens, state_in="fp32", state_out="fp32", seed=31)
    x = make_inputs(w, device="cuda")

    def call(q, k, v, g, beta):
        out, fin = torch.zeros_like(x["v"]), torch.zeros_like(x["final_state"])
        F.fwd(q, k, v, g, beta, x["scale"], out, x["A_log"], x["dt_bias"], x["lower_bound"], initial_state=x["initial_state"],
              final_state=fin, cu_seqlens=x["cu_seqlens"], flags=F.FLAG_NO_FUSED_SHORT)
        return out, fin

    out, fin = call(*(x[n] for n in ("q", "k", "v", "g", "beta")))
    ends = [sum(lens[:i]) for i in range(len(lens) + 1)]
    for spoilt in (0, 1):
        bad = {n: x[n].clone() for n in ("q", "k", "v", "g", "beta")}
        for i in range(spoilt, len(lens), 2):
            for n in bad:
                bad[n][:, ends[i]:ends[i + 1]] = float("nan") if i % 4 < 2 else float("inf")
        o, f = call(*bad.values())
        for i in range(1 - spoilt, len(lens), 2):
            assert torch.equal(o[:, ends[i]:ends[i + 1]].view(torch.int16), out[:, ends[i]:ends[i + 1]].view(torch.int16)), (spoilt, i)
            assert torch.equal(f[i], fin[i]), (spoilt, i)


@pytest.mark.parametrize("T", [64, 75])
def test_gate_parameters_at_the_ends_of_their_range(T):
    """A gate whose slope underflows or overflows and biases that saturate it, in whole chunks and in the last one of a sequence
    (whose absent tokens the kernel stands for by a gate input of minus infinity)."""
    w = Workload("e", H=4, T=T, state_in="fp32", state_out="fp32", seed=32)
    x = make_inputs(w)
    x["A_log"] = torch.tensor([-100.0, 60.0, 1.0, 0.0])
    x["dt_bias"][2, ::2] = 1e30
    x["dt_bias"][2, 1::2] = -1e30
    x["dt_bias"][3, ::2] = float("inf")
    x["dt_bias"][3, 1::2] = -float("inf")
    xc = to_cuda(x)
    out, fin = torch.full_like(xc["v"], float("nan")), torch.full_like(xc["final_state"], float("nan"))
    F.fwd(xc["q"], xc["k"], xc["v"], xc["g"], xc["beta"], x["scale"], out, xc["A_log"], xc["dt_bias"], x["lower_bound"],
          initial_state=xc["initial_state"], final_state=fin)
    o64, s64 = oracle.recurrence_f64(x["q"], x["k"], x["v"], x["g"], x["beta"], x["scale"], x["A_log"], x["dt_bias"], x["lower_bound"],
                                     initial_state=x["initial_state"])
    assert max_abs(out.cpu(), o64) <= OUT_MAX_ABS
    for h in range(4):
        assert rel_fro(fin.cpu()[:, h], s64[:, h]) <= STATE_REL, h


@pytest.mark.parametrize("state", [None, "bf16", "fp32"])
@pytest.mark.parametrize("packed", [False, True], ids=["equal", "packed"])
@pytest.mark.parametrize("lasting", ["all", "none", "first", "odd", "pairs"])
def test_runs_whose_maps_last_or_vanish(lasting, packed, state):
    """The transition map of a run is found to be zero, or is chained: runs of tokens without any decay (the state at their start
    reaches through them) among runs with ordinary gates, in every order; the packed batch has an empty sequence and one shorter
    than the runs."""
    H, lens = 2, [32 * 200 + 9, 0, 32 * 180, 32 * 3 + 1] if packed else None
    w = Workload("m", H=H, T=0 if packed else 32 * 200 + 9, seq_lens=lens, state_in=state, state_out=state or "fp32", state_std=0.5, seed=61, lower_bound=-2.0)
    chunks = (sum(lens) * 4 // (len(lens) * 3) if packed else w.T) // 32 + 1
    average = (sum(lens) // len(lens) if packed else w.T) // 32 + 1
    runs = min(F.plan_segments(w.N * H, chunks)[0], F.plan_segments(w.N * H, average)[0])
    assert runs >= 5
    x = make_inputs(w)
    ends = [sum(lens[:i]) for i in range(len(lens) + 1)] if packed else [0, w.T]
    per = 32 * max(8, -(-(200 + 1) // runs))
    chosen = {"all": lambda r: True, "none": lambda r: False, "first": lambda r: r == 0, "odd": lambda r: r % 2 == 1, "pairs": lambda r: r % 4 >= 2}[lasting]
    for a, b in zip(ends, ends[1:]):
        for r in range(runs):
            if chosen(r):
                x["g"][:, min(a + r * per, b):min(a + (r + 1) * per, b)] = -12.0
    x["A_log"].fill_(0.5)
    xc = to_cuda(x)
    out, fin = torch.full_like(xc["v"], float("nan")), torch.full_like(xc["final_state"], float("nan"))
    ws = torch.empty(F.get_workspace_size(x["q"].shape[1], H, w.N), dtype=torch.uint8, device="cuda")
    for _ in range(2):
        F.fwd(xc["q"], xc["k"], xc["v"], xc["g"], xc["beta"], x["scale"], out, xc["A_log"], xc["dt_bias"], x["lower_bound"],
              initial_state=xc["initial_state"], final_state=fin, cu_seqlens=xc["cu_seqlens"], workspace=ws)
        assert F.read_status(ws) == 0
        ws.fill_(0xFF)                   # (not-a-number in whatever the second call should not read)
    o64, s64 = oracle.recurrence_f64(x["q"], x["k"], x["v"], x["g"], x["beta"], x["scale"], x["A_log"], x["dt_bias"], x["lower_bound"],
                                     initial_state=x["initial_state"], cu_seqlens=x["cu_seqlens"])
    assert max_abs(out.cpu(), o64) <= OUT_MAX_ABS and rel_fro(out.cpu(), o64) <= 1e-2
    assert rel_fro(fin.cpu(), s64) <= STATE_REL


@pytest.mark.parametrize("lasting", ["all", "none", "odd"])
@pytest.mark.parametrize("H,T,beside", [(1, 32 * 100 + 1, True), (4, 32 * 128, True), (16, 32 * 256, False)])
def test_maps_and_offsets_beside_one_another_and_in_turn(H, T, beside, lasting):
    """The first pass over runs, with M and N of a run in two CTAs of a cluster where all of them are resident at once, else in turn in one."""
    w = Workload("b", H=H, T=T, state_in="fp32", state_out="fp32", state_std=0.5, seed=T + H, lower_bound=-2.0)
    runs, length = F.plan_segments(H, (T + 31) // 32)
    assert runs > 2 and (H * (runs - 1) * 2 <= torch.cuda.get_device_properties(0).multi_processor_count) == beside
    x = make_inputs(w)
    for r in range(runs):
        if lasting == "all" or (lasting == "odd" and r % 2 == 1):
            x["g"][:, r * length * 32:(r + 1) * length * 32] = -12.0
    x["A_log"].fill_(0.5)
    xc = to_cuda(x)
    ws = torch.full((F.get_workspace_size(T, H, 1),), 0xFF, dtype=torch.uint8, device="cuda")
    F.fwd(xc["q"], xc["k"], xc["v"], xc["g"], xc["beta"], x["scale"], xc["out"], xc["A_log"], xc["dt_bias"], x["lower_bound"],
          initial_state=xc["initial_state"], final_state=xc["final_state"], workspace=ws)
    assert F.read_status(ws) == 0
    o64, s64 = oracle.recurrence_f64(x["q"], x["k"], x["v"], x["g"], x["beta"], x["scale"], x["A_log"], x["dt_bias"], x["lower_bound"],
                                     initial_state=x["initial_state"])
    assert max_abs(xc["out"].cpu(), o64) <= OUT_MAX_ABS and rel_fro(xc["out"].cpu(), o64) <= 1e-2
    assert rel_fro(xc["final_state"].cpu(), s64) <= STATE_REL


@pytest.mark.parametrize("where", ["state", "v", "k", "g", "beta", "q"])
@pytest.mark.parametrize("value", [float("nan"), float("inf")], ids=["nan", "inf"])
@pytest.mark.parametrize("lens,state", [((16384,), "fp32"), ((9000, 3000, 3), "fp32"), ((6400, 6400), "bf16")], ids=["equal", "packed", "packed_bf16"])
def test_not_a_number_reaches_to_the_end_of_a_sequence_cut_into_runs(lens, state, value, where):
    """With gates that forget everything within a run: what is not finite reaches as far as in the walk of a whole sequence, which
    runs that start from a vanished map would cut short.  Everything else is as close as the two forms are."""
    H = 2
    w = Workload("nan", H=H, seq_lens=list(lens), state_in=state, state_out=state, seed=91)
    x = make_inputs(w, device="cuda")
    assert F.plan_segments(len(lens) * H, (sum(lens) // len(lens) + 31) // 32)[0] > 1
    if where == "state":
        x["initial_state"][0, 0, 5, 7] = value
        x["initial_state"][len(lens) - 1, 1, 100, 3] = value
    elif where == "beta":
        x["beta"][0, 2100, 1] = value if value != value else -value       # (sigmoid(inf) is a number)
    else:
        x[where][0, 700, 0, 33] = value
        x[where][0, 5000, 1, 4] = value
    inputs = {n: x[n] for n in ("q", "k", "v", "g", "beta")}
    common = (x["A_log"], x["dt_bias"], x["lower_bound"])
    packed = x["cu_seqlens"] if len(lens) > 1 else None
    F.fwd(*inputs.values(), x["scale"], x["out"], *common, initial_state=x["initial_state"], final_state=x["final_state"], cu_seqlens=packed)
    a = 0
    for n, length in enumerate(lens):
        part = {name: t[:, a:a + length].contiguous() for name, t in inputs.items()}
        out, fin = torch.empty_like(part["v"]), torch.empty_like(x["final_state"][n:n + 1])
        F.fwd(*part.values(), x["scale"], out, *common, initial_state=x["initial_state"][n:n + 1], final_state=fin, flags=F.FLAG_SCAN_NO_SEGMENTS)
        for got, want in ((x["out"][:, a:a + length], out), (x["final_state"][n:n + 1], fin)):
            finite = torch.isfinite(want)
            assert torch.equal(torch.isfinite(got), finite), (n, int((torch.isfinite(got) != finite).sum()))
            assert not finite.any() or max_abs(got[finite], want[finite]) <= OUT_MAX_ABS
        a += length


def test_the_longest_sequence_of_a_skewed_batch_sets_the_time():
    """Persistent recurrence: the walks are handed out longest first, and a CTA takes its next one near the end of its walk.  Taken with
    the first items, one of four sequences of 200 chunks waits behind the one of 512 on the same SM: 712 chunks instead of 512
    (measured 843 us against 621 for the longest alone; now 626).  The bound lies halfway between the two: 1 + 200 / 512 / 2."""
    def stage_time(lens):
        w = Workload("skew", H=32, seq_lens=lens, state_out="fp32", seed=8)
        x = make_inputs(w, device="cuda")
        args = (x["q"], x["k"], x["v"], x["g"], x["beta"], x["scale"], x["out"], x["A_log"], x["dt_bias"], x["lower_bound"])
        ws = torch.empty(F.get_workspace_size(sum(lens), w.H, w.N), dtype=torch.uint8, device="cuda")
        F.operands(*args, cu_seqlens=x["cu_seqlens"], workspace=ws)
        times = []
        for _ in range(9):
            begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            begin.record()
            F.recurrence(*args, final_state=x["final_state"], cu_seqlens=x["cu_seqlens"], workspace=ws)
            end.record()
            torch.cuda.synchronize()
            times.append(begin.elapsed_time(end))
        return sorted(times)[len(times) // 2]

    alone, skewed = stage_time([16384] + [64] * 124), stage_time([16384] + [6400] * 4 + [64] * 60)
    print(f"longest alone {alone:.3f} ms, skewed {skewed:.3f} ms")
    assert skewed <= alone * 1.195


@pytest.mark.parametrize("T,asks", [(1, 0), (4, 0), (5, 1), (40, 1)])
def test_a_decode_step_asks_for_no_scratch_memory(T, asks):
    w = Workload("d", H=4, B=3, T=T, state_in="fp32", state_out="fp32", seed=T)
    x = make_inputs(w, device="cuda")
    call = lambda: F.fwd(x["q"], x["k"], x["v"], x["g"], x["beta"], x["scale"], x["out"], x["A_log"], x["dt_bias"], x["lower_bound"],
                         initial_state=x["initial_state"], final_state=x["final_state"])
    call()
    torch.cuda.synchronize()
    before = torch.cuda.memory_stats()["allocation.all.allocated"]
    call()
    assert torch.cuda.memory_stats()["allocation.all.allocated"] - before == asks
