"""The calls of `flash_kda.fwd` whose speed matters, over the range a user makes them.

A case is one forward pass of the operator: `B` sequences of `T` tokens, or (`n_seqs` > 0) a packed batch described by
`cu_seqlens`, with `H` heads of 128 channels.  Inputs are the synthetic tensors of `flashkda_b200.workloads` (unit normal
q, k, v, g, beta logits; A_log = log U(1, 16); dt_bias of 0.1; states of 0.02), which are those of the benchmark and of the
parity tests.  Sizes come from the benchmark's configurations and from the tests, or lie between them.

Every call goes through the drop-in signature with nothing else kept: like a user's program, it leaves the scratch memory to
the operator.
"""
import math
import random

import torch

import flash_kda
from flashkda_b200.workloads import D, Workload, algorithmic_bytes, make_inputs

# Token-heads of the largest listed case (C2, 120 206 tokens x 32 heads); a drawn case has no more.
MOST_TOKEN_HEADS = 120206 * 32
MOST_CHAINS = 16384           # states of a batch: 64 KB each in fp32


def _case(H, B=1, T=0, n_seqs=0, n_single=0, lo=0, hi=0, len_seed=0, state_in=None, state_out=None, lower_bound=-5.0):
    """Fixed length: B sequences of T tokens.  Packed: `n_seqs` sequences of lo..hi tokens (uniform, from `len_seed`), behind
    `n_single` sequences of one token."""
    return dict(H=H, B=B, T=T, n_seqs=n_seqs, n_single=n_single, lo=lo, hi=hi, len_seed=len_seed,
                state_in=state_in, state_out=state_out, lower_bound=lower_bound)


def _lengths(case):
    """Sequence lengths of a packed batch, or None for equal lengths."""
    if case["n_seqs"] == 0:
        return None
    gen = torch.Generator().manual_seed(case["len_seed"])
    drawn = torch.randint(case["lo"], case["hi"] + 1, (case["n_seqs"],), generator=gen).tolist()
    return [1] * case["n_single"] + drawn


def _sizes(case):
    """(tokens in all, sequences)"""
    lens = _lengths(case)
    return (case["B"] * case["T"], case["B"]) if lens is None else (sum(lens), len(lens))


def listed():
    return [
        # one decode step of one request: nothing but latency
        dict(_case(32, B=1, T=1, state_in="fp32", state_out="fp32"), name="decode_b1"),
        # one speculative step of a serving batch: a few tokens each, half-precision states
        dict(_case(32, B=64, T=5, state_in="bf16", state_out="bf16"), name="step_b64_t5"),
        # the benchmark's short continuation: state traffic sets the time
        dict(_case(32, B=512, T=16, state_in="fp32", state_out="fp32"), name="continue_b512_t16"),
        # the benchmark's smallest prefill, a few heads of one short prompt
        dict(_case(4, B=1, T=1024, state_out="fp32"), name="prompt_t1024_h4"),
        # an ordinary prompt of odd length on all heads
        dict(_case(32, B=1, T=777, state_out="bf16"), name="prompt_t777_h32"),
        # a batch of medium prompts, more (sequence, head) chains than the chip has processors
        dict(_case(12, B=24, T=1000, state_in="fp32", state_out="fp32"), name="batch_b24_t1000_h12"),
        # the benchmark's headline: fixed-length prefill
        dict(_case(32, B=4, T=8192, state_in="fp32", state_out="fp32"), name="prefill_b4_t8192_h32"),
        # one long prompt on many heads, no state in or out
        dict(_case(96, B=1, T=8192), name="prefill_t8192_h96"),
        # one processor's share of the long-context configuration: few heads, one very long sequence
        dict(_case(8, B=1, T=131072, state_in="fp32", state_out="fp32", lower_bound=-2.0), name="long_t131072_h8"),
        # the benchmark's packed prefill, lengths U[256, 16384]
        dict(_case(32, n_seqs=16, lo=256, hi=16384, state_in="bf16", state_out="bf16"), name="packed_n16_h32"),
        # many short ragged sequences in one packed batch
        dict(_case(16, n_seqs=200, lo=1, hi=300, len_seed=5, state_in="fp32", state_out="fp32"), name="packed_n200_short_h16"),
        # a serving step that mixes decode tokens of running requests with the prompts of new ones
        dict(_case(32, n_seqs=4, n_single=96, lo=500, hi=4000, len_seed=7, state_in="bf16", state_out="bf16"), name="packed_mixed_h32"),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng: random.Random):
    """One more call of the same kinds: steps of a few tokens, equal-length prefills, long sequences on few heads, packed
    batches, packed batches with decode tokens; sizes log-uniform, odd ones included."""
    kind = rng.choice(["step", "prefill", "prefill", "long", "packed", "packed_short", "mixed"])
    H = rng.choice([1, 2, 3, 4, 6, 8, 12, 16, 24, 32, 48, 64, 96])
    state = rng.choice([(None, None), (None, "fp32"), (None, "bf16"), ("fp32", "fp32"), ("fp32", "fp32"), ("bf16", "bf16")])
    bound = rng.choice([-5.0, -5.0, -2.0, -1.0])
    more = dict(state_in=state[0], state_out=state[1], lower_bound=bound)
    if kind == "step":
        state = rng.choice([("fp32", "fp32"), ("bf16", "bf16")])
        more.update(state_in=state[0], state_out=state[1])
        return _case(H, B=_log_int(rng, 1, min(512, MOST_CHAINS // H)), T=rng.randint(1, 32), **more)
    if kind == "prefill":
        T = _log_int(rng, 33, 16384)
        return _case(H, B=_log_int(rng, 1, max(1, min(64, MOST_TOKEN_HEADS // 2 // (T * H)))), T=T, **more)
    if kind == "long":
        H = rng.choice([1, 2, 4, 8, 16])
        return _case(H, B=1, T=_log_int(rng, 16384, min(131072, MOST_TOKEN_HEADS // H)), **more)
    seed = rng.randrange(1 << 20)
    if kind == "packed":
        hi = _log_int(rng, 512, 16384)
        n = _log_int(rng, 2, max(2, min(64, MOST_TOKEN_HEADS // (hi * H))))
        return _case(H, n_seqs=n, lo=hi // 64, hi=hi, len_seed=seed, **more)
    if kind == "packed_short":
        hi = _log_int(rng, 32, 512)
        n = _log_int(rng, 16, max(16, min(512, MOST_CHAINS // H, MOST_TOKEN_HEADS // (hi * H))))
        return _case(H, n_seqs=n, lo=1, hi=hi, len_seed=seed, **more)
    hi = _log_int(rng, 256, 8192)
    n = rng.randint(1, max(1, min(8, MOST_TOKEN_HEADS // (hi * H) - 1)))
    return _case(H, n_seqs=n, n_single=_log_int(rng, 4, min(256, MOST_CHAINS // H)), lo=hi // 8, hi=hi, len_seed=seed, **more)


def prepare(case, seed):
    """The inputs of one call and the tensors its results go to."""
    w = Workload("case", H=case["H"], B=case["B"], T=case["T"], seq_lens=_lengths(case), lower_bound=case["lower_bound"],
                 state_in=case["state_in"], state_out=case["state_out"], seed=seed)
    return make_inputs(w, device="cuda")


def run(x):
    flash_kda.fwd(x["q"], x["k"], x["v"], x["g"], x["beta"], x["scale"], x["out"], x["A_log"], x["dt_bias"], x["lower_bound"],
                  initial_state=x["initial_state"], final_state=x["final_state"], cu_seqlens=x["cu_seqlens"])
    return {"out": x["out"], "final_state": x["final_state"]}


def work(case):
    """Bytes: every input read once, every output written once.  Operations: those of the per-token recurrence (k S, the
    rank-one update and q S, a multiply and an add per state element each); chunked forms need no fewer."""
    tokens, n = _sizes(case)
    return {"bytes": algorithmic_bytes(tokens, case["H"], n, case["state_in"], case["state_out"]),
            "flops": 6 * D * D * tokens * case["H"]}


def tolerance(case):
    # bf16 operands and bf16 results throughout, fp32 accumulation (fp32 states carry the operands' bf16 rounding too)
    return {"rel": 1e-2}
