"""The work this framework is used for, as cases that can be timed and compared.

Four kinds of call, each through the public entry points:

  train    `naju_scan` and its backward: one scan of a training step, all gradients
  prefill  `naju_scan` without gradients, final state returned: a prompt (or the next piece of one)
  decode   `naju_scan_step` once per layer of a stack: one token for every sequence of the batch
  host     `scan_fwd_bwd_host`: forward and backward of tensors that live in pinned host memory

Data types (`dtype`): "bf16" activations, logits and B / C; "mixed" bf16 with fp32 logits, what a mixer
hands over under bf16 autocast; "f16"; "f32".  `mixer` true: u is time-contiguous (a depthwise convolution's
output seen as [B, T, D]) and B, C are the two halves of one [B, T, 2N] tensor.  `carry` true: an initial state
is given and the final one returned.  `skip` true: D_skip is not zero.  `f_mean`, `i_mean`: where the normal
distributions of the retention and write logits are centred.
"""
import torch

from naju_b200 import naju_scan, naju_scan_step, scan_fwd_bwd_host

_TYPES = {"bf16": (torch.bfloat16, torch.bfloat16), "mixed": (torch.bfloat16, torch.float32),
          "f16": (torch.float16, torch.float16), "f32": (torch.float32, torch.float32)}


def _scan(op, B, T, D, N, dtype, f_mean=2.0, i_mean=0.0, mixer=False, carry=False, skip=False):
    return {"op": op, "B": B, "T": T, "D": D, "N": N, "dtype": dtype, "f_mean": f_mean, "i_mean": i_mean,
            "mixer": mixer, "carry": carry, "skip": skip}


def _decode(layers, B, D, N, dtype):
    return {"op": "decode", "layers": layers, "B": B, "D": D, "N": N, "dtype": dtype}


def listed():
    return [
        # the smallest training call: launches and the host path are all of it
        dict(_scan("train", 2, 512, 64, 16, "f32"), name="train_small_f32"),
        # full-precision training at an ordinary size
        dict(_scan("train", 4, 2048, 1024, 16, "f32", skip=True), name="train_f32"),
        # a short batch padded to its longest sequence, whose length is no multiple of anything
        dict(_scan("train", 3, 1021, 1536, 16, "bf16", skip=True), name="train_ragged"),
        # one mixer layer of a model with d_model 1024, as the mixer hands its tensors over
        dict(_scan("train", 8, 4096, 2048, 16, "mixed", f_mean=5.0, i_mean=-2.0, mixer=True), name="train_mixer_layer"),
        # the benchmark's configuration
        dict(_scan("train", 8, 16384, 2048, 16, "bf16"), name="train_long_batch"),
        # long sequences with retention close to one
        dict(_scan("train", 4, 65536, 2048, 16, "bf16", f_mean=4.0), name="train_long_sequence"),
        # wide model, 64 states: one GPU's part of the large-batch configuration
        dict(_scan("train", 8, 8192, 4096, 64, "bf16"), name="train_wide_state"),
        # one prompt
        dict(_scan("prefill", 1, 4096, 2048, 16, "mixed", f_mean=5.0, i_mean=-2.0, mixer=True), name="prefill_one"),
        # the next piece of many prompts, from the states that the piece before left
        dict(_scan("prefill", 16, 1024, 2048, 16, "bf16", carry=True), name="prefill_batch_carried"),
        # one sequence decoded by a 24-layer stack
        dict(_decode(24, 1, 2048, 16, "bf16"), name="decode_one"),
        # the decode configuration: 256 sequences
        dict(_decode(24, 256, 2048, 16, "bf16"), name="decode_batch"),
        # activations off-loaded to the host
        dict(_scan("host", 8, 2048, 2048, 16, "bf16"), name="host_rows"),
    ]


def _between(rng, lo, hi):
    """A whole number from lo to hi, spread evenly over its logarithm."""
    return min(hi, max(lo, int(round(lo * (hi / lo) ** rng.random()))))


_MOST_CHANNEL_STEPS = 8 * 8192 * 4096  # the wide-state case's


def _padded(N):
    return 16 if N <= 16 else 32 if N <= 32 else 64 if N <= 64 else 128


def draw(rng):
    op = rng.choice(["train"] * 5 + ["prefill"] * 2 + ["decode"] * 2 + ["host"])
    # channels: a multiple of 64 as model widths are, at times of 8, seldom any number
    step = rng.choice([64, 64, 64, 64, 8, 1])
    if op == "decode":
        D = max(step, _between(rng, 256, 4096) // step * step)
        N = rng.choice([16, 16, 16, 8, 32, 64])
        return _decode(rng.choice([12, 24]), _between(rng, 1, 256), D, N, rng.choice(["bf16", "bf16", "mixed", "f16", "f32"]))
    if op == "host":
        return _scan(op, _between(rng, 2, 8), _between(rng, 256, 2048), max(step, _between(rng, 256, 2048) // step * step),
                     16, rng.choice(["bf16", "mixed", "f32"]))
    D = max(step, _between(rng, 64, 4096) // step * step)
    N = rng.choice([16, 16, 16, 16, 8, 32, 64, rng.randint(1, 64)])
    B, T = _between(rng, 1, 32), _between(rng, 64, 65536)
    if rng.random() < 0.5:
        T = max(64, T // 64 * 64)
    most = _MOST_CHANNEL_STEPS * 64 // max(64, _padded(N))
    while B * T * D > most:
        if B > 1:
            B = max(1, B // 2)
        else:
            T = max(64, T // 2)
    dtype = rng.choice(["bf16", "bf16", "bf16", "mixed", "mixed", "f16", "f32"])
    mixer = dtype == "mixed" and rng.random() < 0.7
    f_mean, i_mean = rng.choice([(2.0, 0.0), (2.0, 0.0), (4.0, 0.0), (5.0, -2.0)])
    return _scan(op, B, T, D, N, dtype, f_mean, i_mean, mixer, rng.random() < 0.3, not mixer and rng.random() < 0.4)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    act, gate = _TYPES[case["dtype"]]

    def normal(*shape, mean=0.0, std=1.0, dtype=torch.float32):
        return torch.randn(*shape, device="cuda", generator=gen).mul_(std).add_(mean).to(dtype)

    B, D, N = case["B"], case["D"], case["N"]
    if case["op"] == "decode":
        L = case["layers"]
        h = normal(L, B, D, N)
        ins = [normal(L, B, D, dtype=act), normal(L, B, D, mean=2.0, dtype=gate), normal(L, B, D, dtype=gate),
               normal(L, B, N, std=N ** -0.5, dtype=act), normal(L, B, N, std=N ** -0.5, dtype=act), normal(L, D, std=0.1)]
        layers = [tuple(t[k] for t in [h] + ins) for k in range(L)]
        return {"case": case, "h": h, "layers": layers}
    T = case["T"]
    if case["mixer"]:
        u = normal(B, D, T, dtype=act).transpose(1, 2)
        Bm, Cm = normal(B, T, 2 * N, std=N ** -0.5, dtype=act).split([N, N], dim=-1)
    else:
        u = normal(B, T, D, dtype=act)
        Bm, Cm = (normal(B, T, N, std=N ** -0.5, dtype=act) for _ in range(2))
    fl = normal(B, T, D, mean=case["f_mean"], dtype=gate)
    il = normal(B, T, D, mean=case["i_mean"], dtype=gate)
    skip = normal(D, std=0.1) if case["skip"] else torch.zeros(D, device="cuda")
    state = {"case": case, "ins": [u, fl, il, Bm, Cm, skip], "h0": normal(B, D, N) if case["carry"] else None}
    if case["op"] in ("train", "host"):
        state["dy"] = normal(B, T, D, dtype=act)
    if case["op"] == "train":
        state["dh"] = normal(B, D, N, std=0.1) if case["carry"] else None
        for t in state["ins"]:
            t.requires_grad_(True)
    if case["op"] == "host":
        pin = lambda t: t.cpu().pin_memory()  # noqa: E731
        state["ins"], state["dy"] = [pin(t) for t in state["ins"]], pin(state["dy"])
        like = lambda t: torch.empty(t.shape, dtype=t.dtype).pin_memory()  # noqa: E731
        hu, hf, hi, hB, hC, hD = state["ins"]
        state["out"] = {"y": like(hu), "du": like(hu), "dfl": like(hf), "dil": like(hi), "dB": like(hB), "dC": like(hC),
                        "dD": like(hD)}
    return state


def run(state):
    op = state["case"]["op"]
    if op == "decode":
        return {"y": [naju_scan_step(*layer)[0] for layer in state["layers"]], "h": state["h"]}
    ins = state["ins"]
    if op == "host":
        return scan_fwd_bwd_host(*ins, state["dy"], rows_per_chunk=1, time_splits=2, out=state["out"])
    if op == "prefill":
        with torch.no_grad():
            return naju_scan(*ins, h0=state["h0"], return_final_state=True)
    if state["h0"] is None:
        y = naju_scan(*ins)
        return [y.detach(), torch.autograd.grad(y, ins, state["dy"])]
    # the carried state is the detached end of the piece before; the next piece's adjoint comes back into this one
    y, h = naju_scan(*ins, h0=state["h0"], return_final_state=True)
    return [y.detach(), h.detach(), torch.autograd.grad([y, h], ins, [state["dy"], state["dh"]])]


def work(case):
    """Every tensor of a call once.  A training pass is two calls, the backward after the forward has returned, so
    what both need counts in both; a host pass brings its inputs over once and its results back once."""
    B, D, N, op = case["B"], case["D"], case["N"], case["op"]
    act, gate = (torch.finfo(t).bits // 8 for t in _TYPES[case["dtype"]])
    if op == "decode":
        tok = case["layers"] * B
        return {"bytes": tok * (D * (8 * N + 2 * act + 2 * gate) + 2 * N * act) + case["layers"] * D * 4, "flops": tok * D * (5 * N + 10)}
    tok, state = B * case["T"], 4 * B * D * N
    fwd = tok * (D * (2 * act + 2 * gate) + 2 * N * act) + 4 * D
    bwd = tok * (D * (3 * act + 4 * gate) + 4 * N * act) + 8 * D
    fwd += state * (op == "prefill" or case["carry"]) + state * case["carry"]
    bwd += 2 * state * case["carry"]
    fwd_flops, bwd_flops = tok * D * (5 * N + 10), tok * D * (14 * N + 20)
    if op == "prefill":
        return {"bytes": fwd, "flops": fwd_flops}
    if op == "host":
        return {"bytes": tok * (D * (4 * act + 4 * gate) + 4 * N * act) + 8 * D, "flops": fwd_flops + bwd_flops}
    return {"bytes": fwd + bwd, "flops": fwd_flops + bwd_flops}


def tolerance(case):
    # fp32 sums over time, states and channels; results rounded to 16 bits differ by single roundings
    return {"rel": 1e-5} if case["dtype"] == "f32" else {"rel": 4e-3} if case["dtype"] != "f16" else {"rel": 1e-3}
