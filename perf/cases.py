"""The sampling work that a program hands to this library, as a list of timed cases.

Every case goes through the public calls of `born_b200.Sampler`.  A *kind* is the call that is
made:

  sample    one `Sampler.sample` per step into output tensors that the program keeps
  prepared  a decode loop over fixed buffers: `Sampler.prepare` once, `PreparedCall.run` per step
  next      the generate loop: `Sampler.sample_next` over the device-resident token history
  verify    `Sampler.spec_verify` of a draft
  host      `Sampler.sample` on numpy arrays: copied in, sampled, copied out

Sizes are those of the benchmark configurations and of the tests; logits are N(0, s^2), with a
Zipf-shaped bias over a random ranking of the vocabulary where the configuration has one.
"""
import numpy as np
import torch

from born_b200 import Sampler, SamplingConfig
from born_b200.sampler import row_params_array

_DEFAULTS = dict(kind="sample", batch=1, vocab=32000, dtype="f32", history=0, mask=False, segments=0, draft=0,
                 logits="normal", rows="same", temperature=0.0, top_k=0, top_p=0.0, min_p=0.0, repetition=0.0,
                 frequency=0.0, presence=0.0)


def _case(**kw):
    return {**_DEFAULTS, **kw}


def listed():
    return [
        # one user, one token: the smallest call, all latency
        _case(name="single_row", vocab=32000, history=64, logits="spiked", temperature=0.8, top_k=40, top_p=0.95,
              repetition=1.1),
        # a generate loop of a few users on bf16 logits with the history kept on the device
        _case(name="loop_b8", kind="next", batch=8, vocab=128256, dtype="bf16", history=512, logits="zipf",
              temperature=0.8, top_k=50, top_p=0.95, repetition=1.1),
        # host buffers in and out, the form that a program without a GPU tensor type binds
        _case(name="host_b4", kind="host", batch=4, vocab=32000, temperature=0.8, top_k=40, top_p=0.95),
        # an odd batch of an odd vocabulary: rows start at any alignment
        _case(name="ragged_b37", batch=37, vocab=50257, dtype="bf16", temperature=0.9, top_k=50, top_p=0.9),
        # continuous batching, moderate and full batch, with penalties over the prompt and the text so far
        _case(name="decode_b64", kind="prepared", batch=64, vocab=128256, history=512, logits="zipf", temperature=0.7,
              min_p=0.05, top_p=0.9, frequency=0.5, presence=0.3),
        _case(name="decode_b256", kind="prepared", batch=256, vocab=128256, history=512, logits="zipf",
              temperature=0.7, min_p=0.05, top_p=0.9, frequency=0.5, presence=0.3),
        # the common top-k + nucleus setting
        _case(name="topk_b256", batch=256, vocab=128256, logits="zipf", temperature=0.7, top_k=50, top_p=0.9),
        # plain softmax sampling over the whole vocabulary, as training rollouts want it
        _case(name="temperature_b256", batch=256, vocab=128256, logits="zipf", temperature=0.8),
        # nucleus sampling alone, whose nucleus may be any size
        _case(name="top_p_b64", batch=64, vocab=128256, logits="zipf", temperature=0.7, top_p=0.9),
        # grammar-constrained decoding, greedy and sampled rows in one batch
        _case(name="constrained_b256", batch=256, vocab=151936, dtype="bf16", mask=True, logits="grammar",
              rows="alternate", temperature=1.0, top_k=50),
        # speculative decoding: verify five draft tokens of 32 sequences
        _case(name="verify_b32", kind="verify", batch=32, vocab=128256, draft=5, temperature=1.0),
        # the vocab-sharded algorithm on one GPU, at its full batch and vocabulary
        _case(name="segments_b1024", batch=1024, vocab=256000, dtype="bf16", segments=8, logits="spikes",
              temperature=1.0, top_k=64, top_p=0.95),
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def _draw_vocab(rng, lo, hi):
    """Log-uniform; two in three a multiple of 64, as vocabularies are padded to, the others as they fall."""
    v = _log_int(rng, lo, hi)
    return v if rng.random() < 0.34 else max(64, v // 64 * 64)


def draw(rng):
    what = rng.choice(["single", "loop", "host", "decode", "top_k", "temperature", "top_p", "constrained", "verify",
                       "segments", "greedy"])
    dtype = rng.choice(["f32", "bf16"])
    t = round(rng.uniform(0.5, 1.2), 3)
    if what == "single":
        return _case(batch=rng.randint(1, 4), vocab=_draw_vocab(rng, 1000, 262144), dtype=dtype,
                     history=_log_int(rng, 1, 1024), logits="spiked", temperature=t, top_k=rng.randint(10, 100),
                     top_p=0.95, repetition=1.1)
    if what == "loop":
        return _case(kind="next", batch=_log_int(rng, 1, 128), vocab=_draw_vocab(rng, 8192, 200000), dtype=dtype,
                     history=_log_int(rng, 16, 1024), logits="zipf", temperature=t, top_k=rng.randint(20, 100),
                     top_p=0.95, repetition=1.1)
    if what == "host":
        return _case(kind="host", batch=_log_int(rng, 1, 16), vocab=_draw_vocab(rng, 1000, 65536), temperature=t,
                     top_k=rng.randint(20, 60), top_p=0.95)
    if what == "decode":
        return _case(kind=rng.choice(["prepared", "sample"]), batch=_log_int(rng, 8, 400),
                     vocab=_draw_vocab(rng, 16384, 160000), dtype=dtype, history=_log_int(rng, 16, 1024),
                     logits="zipf", temperature=t, min_p=round(rng.uniform(0.02, 0.2), 3), top_p=0.9, frequency=0.5,
                     presence=0.3)
    if what == "top_k":
        return _case(batch=_log_int(rng, 8, 400), vocab=_draw_vocab(rng, 8192, 160000), dtype=dtype,
                     logits=rng.choice(["zipf", "normal"]), temperature=t, top_k=rng.randint(5, 200),
                     top_p=round(rng.uniform(0.8, 0.98), 3))
    if what == "temperature":
        return _case(batch=_log_int(rng, 4, 300), vocab=_draw_vocab(rng, 8192, 160000), dtype=dtype,
                     logits=rng.choice(["zipf", "normal"]), temperature=t)
    if what == "top_p":
        return _case(batch=_log_int(rng, 1, 64), vocab=_draw_vocab(rng, 8192, 128256), dtype=dtype, logits="zipf",
                     temperature=t, top_p=round(rng.uniform(0.5, 0.95), 3))
    if what == "constrained":
        return _case(batch=_log_int(rng, 8, 300), vocab=_draw_vocab(rng, 32000, 160000), dtype=dtype, mask=True,
                     logits="grammar", rows=rng.choice(["alternate", "same"]), temperature=t,
                     top_k=rng.randint(20, 80))
    if what == "verify":
        return _case(kind="verify", batch=_log_int(rng, 1, 32), vocab=_draw_vocab(rng, 16384, 128256),
                     draft=rng.randint(1, 5), temperature=t)
    if what == "segments":
        g = rng.choice([2, 4, 8])
        return _case(batch=_log_int(rng, 64, 1024), vocab=g * 64 * rng.randint(64, 250000 // (g * 64)), dtype="bf16",
                     segments=g, logits="spikes", temperature=t, top_k=rng.randint(8, 64), top_p=0.95)
    return _case(batch=_log_int(rng, 1, 512), vocab=_draw_vocab(rng, 1000, 128256), dtype=dtype, logits="zipf")


# logits of a row: standard deviation of the normal part, and what is added to it
_SCALE = {"normal": 2.0, "spiked": 2.0, "zipf": 3.0, "grammar": 2.5, "spikes": 2.0}


def _logits(case, g):
    B, V = case["batch"], case["vocab"]
    z = torch.randn((B, V), generator=g, device="cuda") * _SCALE[case["logits"]]
    if case["logits"] == "zipf":  # -1.1 ln(rank) over a random ranking
        rank = torch.argsort(torch.rand((B, V), generator=g, device="cuda"), dim=1)
        z -= 1.1 * torch.log(rank.float() + 1.0)
    elif case["logits"] == "spiked":  # three likely tokens
        at = torch.randint(0, V, (B, 3), generator=g, device="cuda")
        z.scatter_add_(1, at, torch.full((B, 3), 8.0, device="cuda"))
    elif case["logits"] == "spikes":  # one token in a hundred
        z += 6.0 * (torch.rand((B, V), generator=g, device="cuda") < 0.01)
    return z if case["dtype"] == "f32" else z.to(torch.bfloat16)


def _mask(case, g):
    """A grammar's bitmask: one token in twenty allowed, at least one in each row."""
    B, V = case["batch"], case["vocab"]
    words = (V + 31) // 32
    bits = torch.rand((B, words * 32), generator=g, device="cuda") < 0.05
    bits[:, V:] = False
    bits[:, 0] |= ~bits.any(dim=1)
    weight = 2 ** torch.arange(32, device="cuda", dtype=torch.int64)
    word = (bits.view(B, words, 32) * weight).sum(-1)
    return torch.where(word >= 2 ** 31, word - 2 ** 32, word).to(torch.int32)


def _uniforms(shape, g):
    return torch.rand(shape, generator=g, device="cuda").clamp_(max=1.0 - 2.0 ** -24)


def _config(case):
    return SamplingConfig(temperature=case["temperature"], top_k=case["top_k"], top_p=case["top_p"],
                          min_p=case["min_p"], repetition_penalty=case["repetition"],
                          frequency_penalty=case["frequency"], presence_penalty=case["presence"])


def _prepare_verify(case, g):
    B, V, K = case["batch"], case["vocab"], case["draft"]
    target = torch.randn((B, K + 1, V), generator=g, device="cuda") * 2.0
    draft = target[:, :K] + 0.5 * torch.randn((B, K, V), generator=g, device="cuda")
    p = torch.softmax(draft.view(B * K, V) / case["temperature"], dim=-1)
    tokens = torch.multinomial(p, 1, generator=g).view(B, K).to(torch.int32)
    return dict(target=target, draft=draft.contiguous(), tokens=tokens, accept=_uniforms((B, K), g),
                resample=_uniforms((B, K + 1), g))


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    B, V, H = case["batch"], case["vocab"], case["history"]
    state = {"kind": case["kind"], "sampler": Sampler(device=0, max_batch=B, max_vocab=V)}
    if case["kind"] == "verify":
        state.update(_prepare_verify(case, g), temperature=case["temperature"])
        return state
    logits = _logits(case, g)
    kw = dict(uniforms=_uniforms((B,), g), config=_config(case), want_prob=True, want_lse=True)
    if case["mask"]:
        kw["mask"] = _mask(case, g)
    if H:
        history = torch.randint(0, V, (B, H), generator=g, device="cuda", dtype=torch.int32)
        if case["kind"] == "next":
            state["sampler"].history_create(H)
            state["sampler"].history_reset(history)
        else:
            kw["history"] = history
    if case["rows"] == "alternate":
        rows = [SamplingConfig(greedy=True) if b % 2 == 0 else _config(case) for b in range(B)]
        kw["row_params"] = torch.from_numpy(row_params_array(rows).view(np.uint8)).cuda()
        del kw["config"]
    if case["segments"]:
        kw["vocab_segments"] = case["segments"]
    if case["kind"] == "host":
        logits, kw["uniforms"] = logits.cpu().numpy(), kw["uniforms"].cpu().numpy()
    state.update(logits=logits, kw=kw)
    kw["out"] = {}
    if case["kind"] == "prepared":
        state["sampler"].reserve(logits, **kw)
        state["call"] = state["sampler"].prepare(logits, **kw)
    return state


def run(state):
    kind = state["kind"]
    if kind == "prepared":
        return state["call"].run()
    if kind == "verify":
        return state["sampler"].spec_verify(state["target"], state["draft"], state["tokens"], state["accept"],
                                            state["resample"], temperature=state["temperature"])
    if kind == "next":
        return state["sampler"].sample_next(state["logits"], **state["kw"])
    return state["sampler"].sample(state["logits"], **state["kw"])


def work(case):
    """Logits, mask, history and uniforms read once, the outputs written once.  Operations: a comparison and the
    shifted exponential of the log-sum-exp for each logit; where whole distributions are compared or drawn from,
    the exact exponential (about sixteen) as well."""
    B, V = case["batch"], case["vocab"]
    if case["kind"] == "verify":
        K = case["draft"]
        n = B * (2 * K + 1) * V
        return {"bytes": 4 * n + 4 * B * (4 * K + 4), "flops": 18 * n}
    n = B * V
    row = V * (4 if case["dtype"] == "f32" else 2) + 4 * case["history"] + 4 + 16
    if case["mask"]:
        row += 4 * ((V + 31) // 32)
    if case["rows"] == "alternate":
        row += 32
    whole = case["temperature"] > 0 and not case["top_k"] and not case["min_p"]
    return {"bytes": B * row, "flops": n * (20 if whole else 4)}


def tolerance(case):
    """Tokens and statuses are whole numbers and stay the same; probabilities and the log-sum-exp are 32-bit."""
    return {"rel": 1e-5, "differ": 0.0}
