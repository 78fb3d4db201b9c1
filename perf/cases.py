"""Performance cases: what a user of the receiver back end has it do.

Each case is one call (or one captured step) through the package's public
entry points, on data shaped like the traffic it stands for:

* demapping: a packet of a few thousand symbols (the smallest call, bound by
  latency), long streams of square QAM with max-log and exact LLRs, and a
  constellation without per-axis factors;
* decoding: one frame, a batch of short frames, a batch of long frames, a
  long code without circulant blocks, and the sum-product rule;
* encoding a batch of long frames;
* the whole receiver: a captured step over frames of three codes, and a point
  of an error-rate curve (bits, encoder, channel, demapper, decoder, counts).

Codes A, B and C and their waterfalls are those of
``commkit_gb300.workloads``; the DVB-S2 codes and the PON code are the ones
the tests hold.  Inputs are made on the GPU from the seed alone with plain
torch, and the 64-bit values of :func:`exact` with plain torch in float64.
"""

from __future__ import annotations

import functools
import math
from pathlib import Path

import numpy as np
import torch

import commkit_gb300 as ck
from commkit_gb300 import pipeline, workloads

GOLDEN = Path(ck.__file__).resolve().parent.parent / "tests" / "golden"
CODES = ("A", "B", "C", "dvbs2_normal", "dvbs2_short", "pon")
LN2 = math.log(2.0)


def listed() -> list[dict]:
    return [
        # One packet of a burst receiver: the call's own latency.
        dict(name="llr_packet", kind="llr", family="qam", order=16, method="maxlog", symbols=4096, esn0_db=14.0),
        # The demapper at scale: a long 64-QAM capture, max-log.
        dict(name="llr_stream", kind="llr", family="qam", order=64, method="maxlog", symbols=1 << 22, esn0_db=18.0),
        # The same scale with exact log-sum-exp LLRs; an odd count.
        dict(name="llr_exact", kind="llr", family="qam", order=16, method="exact", symbols=(1 << 22) - 1, esn0_db=11.0),
        # Cross QAM has no per-axis factors: every point is measured.
        dict(name="llr_cross", kind="llr", family="qam", order=128, method="maxlog", symbols=1000003, esn0_db=21.0),
        # One short frame: the decoder's latency.
        dict(name="decode_frame", kind="decode", code="A", rule="min_sum", iterations=20, frames=1, ebn0_db=2.5),
        # A batch of short frames above the waterfall (few, uneven iterations).
        dict(name="decode_short", kind="decode", code="A", rule="min_sum", iterations=20, frames=1024, ebn0_db=2.5),
        # A large batch of long frames of the big circulant code.
        dict(name="decode_long", kind="decode", code="C", rule="min_sum", iterations=50, frames=1216, ebn0_db=2.8),
        # A long code whose rows are no circulants: the DVB-S2 normal frame.
        dict(name="decode_dvbs2", kind="decode", code="dvbs2_normal", rule="min_sum", iterations=50, frames=64,
             ebn0_db=1.5),
        # The sum-product rule, for the last tenths of a dB.
        dict(name="decode_sum_product", kind="decode", code="B", rule="sum_product", iterations=20, frames=256,
             ebn0_db=4.0),
        # A transmitter's batch of long frames.
        dict(name="encode_long", kind="encode", code="C", frames=1000),
        # A captured receiver step over mixed traffic of three codes.
        dict(name="receive_mixed", kind="mixed", frames=2048, spread_db=1.0),
        # One point of an error-rate curve at its default batch size.
        dict(name="error_rate_point", kind="curve", code="A", order=4, ebn0_db=2.0, blocks=2000),
    ]  # fmt: skip


def _log_int(rng, low: int, high: int) -> int:
    return min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high + 1))))))


# Per code: the most frames drawn (an eighth of them with sum-product, which
# costs several times more), and the Eb/N0 (dB, binary signalling) range from
# just above its waterfall to a point where it converges in a few iterations.
_FRAMES = {"A": 4096, "B": 2048, "C": 608, "dvbs2_normal": 64, "dvbs2_short": 256, "pon": 192}
_EBN0 = {"A": (2.0, 3.5), "B": (3.8, 5.5), "C": (2.7, 4.0), "dvbs2_normal": (1.5, 2.5), "dvbs2_short": (1.8, 3.0),
         "pon": (4.0, 5.0)}  # fmt: skip


def draw(rng) -> dict:
    """A case of the listed ranges; a drawn case costs no more than the
    largest listed one."""
    kind = rng.choice(["llr", "llr", "llr", "decode", "decode", "decode", "encode", "mixed", "curve"])
    if kind == "llr":
        family, order = rng.choice([("qam", 4), ("qam", 16), ("qam", 64), ("qam", 256), ("qam", 8), ("qam", 32),
                                    ("qam", 128), ("psk", 8), ("psk", 16)])  # fmt: skip
        square = family == "qam" and math.isqrt(order) ** 2 == order
        method = rng.choice(["maxlog", "exact"])
        return dict(kind="llr", family=family, order=order, method=method,
                    symbols=_log_int(rng, 256, 1 << 22 if square else 1 << 20),
                    esn0_db=round(rng.uniform(3.0, 6.0) + 2.6 * math.log2(order), 2))  # fmt: skip
    if kind == "decode":
        rule = rng.choice(["min_sum", "min_sum", "sum_product"])
        code = rng.choice(CODES if rule == "min_sum" else ("A", "B", "dvbs2_short", "pon"))
        frames = _FRAMES[code] // (8 if rule == "sum_product" else 1)
        return dict(kind="decode", code=code, rule=rule, iterations=rng.choice([20, 30, 50]),
                    frames=_log_int(rng, 1, frames), ebn0_db=round(rng.uniform(*_EBN0[code]), 2))  # fmt: skip
    if kind == "encode":
        code = rng.choice(("A", "B", "C", "dvbs2_normal"))
        return dict(kind="encode", code=code, frames=_log_int(rng, 1, 2 * _FRAMES[code]))
    if kind == "mixed":
        return dict(kind="mixed", frames=_log_int(rng, 32, 2048), spread_db=round(rng.uniform(0.2, 1.0), 2))
    code, order = rng.choice([("A", 4), ("A", 16), ("B", 4), ("B", 16)])
    low = 2.0 + (1.5 if code == "B" else 0.0) + (2.5 if order == 16 else 0.0)
    return dict(kind="curve", code=code, order=order, ebn0_db=round(rng.uniform(low, low + 2.0), 2),
                blocks=_log_int(rng, 50, 2000 if code == "A" else 1000))  # fmt: skip


# ---------------------------------------------------------------------------
# What a program keeps: codes and constellations
# ---------------------------------------------------------------------------


@functools.lru_cache(maxsize=None)
def _edges(name: str) -> tuple:
    """(checks, variables, num_checks, num_variables, sent bits) of a code."""
    if name in workloads.CODES:
        spec = workloads.CODES[name]
        checks, variables = workloads.lift(spec.base(), spec.z)
        return checks, variables, spec.mb * spec.z, spec.nb * spec.z, spec.nb * spec.z
    tag, file = {"dvbs2_normal": ("dvbs2n", "dvbs2_normal.npz"), "dvbs2_short": ("dvbs2s", "ldpc_golden.npz"),
                 "pon": ("pon", "ldpc_golden.npz")}[name]  # fmt: skip
    d = np.load(GOLDEN / file)
    m, N, n = (int(d[f"{tag}_{s}"]) for s in ("m", "N", "n"))
    return d[f"{tag}_checks"], d[f"{tag}_variables"], m, N, n


@functools.lru_cache(maxsize=None)
def _code(name: str) -> ck.LDPCCode:
    if name in workloads.CODES:
        spec = workloads.CODES[name]
        return ck.LDPCCode.quasi_cyclic(spec.base(), lifting=spec.z)
    checks, variables, m, N, n = _edges(name)
    return ck.LDPCCode(checks, variables, m, N, N - n)


@functools.lru_cache(maxsize=None)
def _constellation(family: str, order: int) -> ck.Constellation:
    return ck.Constellation.psk(order) if family == "psk" else ck.Constellation.qam(order)


def _method(case: dict):
    rule = ck.MinSum if case["rule"] == "min_sum" else ck.SumProduct
    return rule(max_iterations=case["iterations"])


# ---------------------------------------------------------------------------
# Inputs, made with plain torch on the GPU
# ---------------------------------------------------------------------------


def _generator(seed: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(seed)


@functools.lru_cache(maxsize=None)
def _encoder(name: str) -> tuple:
    """Information edges on the GPU and the accumulator's stride: every listed
    code's parity bit j is its check's information sum plus parity bit
    j - stride."""
    checks, variables, m, N, _ = _edges(name)
    info = variables < N - m
    first = np.sort(checks[variables == N - m])
    stride = int(first[1])
    dev = [torch.from_numpy(a[info].astype(np.int64)).cuda() for a in (checks, variables)]
    return dev[0], dev[1], m, N, stride


def _codewords(name: str, frames: int, gen: torch.Generator) -> torch.Tensor:
    """(frames, N) codewords as int8 (the PON code, whose parity part is no
    accumulator, sends its all-zero codeword)."""
    if name == "pon":
        return torch.zeros((frames, _edges(name)[3]), dtype=torch.int8, device="cuda")
    checks, variables, m, N, g = _encoder(name)
    out = torch.empty((frames, N), dtype=torch.int8, device="cuda")
    for i in range(0, frames, 256):
        u = torch.randint(0, 2, (min(256, frames - i), N - m), device="cuda", generator=gen, dtype=torch.int8)
        s = torch.zeros((u.shape[0], m), device="cuda").index_add_(1, checks, u[:, variables].float())
        p = s.view(-1, m // g, g).cumsum(1).remainder(2.0).view(-1, m)
        out[i : i + 256] = torch.cat([u, p.to(torch.int8)], 1)
    return out


def _binary_llrs(case: dict, seed: int) -> torch.Tensor:
    """Float32 channel LLRs (frames, sent bits) of binary signalling (each
    axis of Gray QPSK) over Gaussian noise at the case's Eb/N0."""
    gen = _generator(seed)
    _, _, m, N, n = _edges(case["code"])
    words = _codewords(case["code"], case["frames"], gen)[:, :n]
    esn0 = 10.0 ** (case["ebn0_db"] / 10.0) * (N - m) / n  # per bit: Es/N0 of one axis
    var = 1.0 / (2.0 * esn0)
    noise = torch.randn(words.shape, device="cuda", generator=gen)
    return (1.0 - 2.0 * words.float() + math.sqrt(var) * noise) * (2.0 / var)


def _map(bits: torch.Tensor, c: ck.Constellation) -> torch.Tensor:
    """(..., n) bits, MSB first, to complex64 symbols (..., n / k)."""
    k = c.bits_per_symbol
    weights = 1 << torch.arange(k - 1, -1, -1, device="cuda")
    label = (bits.view(*bits.shape[:-1], -1, k).long() * weights).sum(-1)
    by_label = np.empty(c.order, np.complex64)
    by_label[(c.bit_labels.astype(np.int64) << np.arange(k - 1, -1, -1)).sum(1)] = c.points
    return torch.from_numpy(by_label).cuda()[label]


def _awgn(x: torch.Tensor, noise_var, gen: torch.Generator) -> torch.Tensor:
    noise = torch.randn((*x.shape, 2), device="cuda", generator=gen)
    return x + torch.view_as_complex(noise) * (noise_var / 2.0) ** 0.5


def _prepare_llr(case: dict, seed: int) -> dict:
    gen = _generator(seed)
    c = _constellation(case["family"], case["order"])
    bits = torch.randint(0, 2, (case["symbols"] * c.bits_per_symbol,), device="cuda", generator=gen)
    noise_var = float(np.mean(np.abs(c.points) ** 2)) / 10.0 ** (case["esn0_db"] / 10.0)
    x = _awgn(_map(bits, c), noise_var, gen).contiguous()
    return dict(symbols=x, noise_var=noise_var, constellation=c, method=case["method"])


def _mixed_inputs(case: dict, seed: int) -> list[tuple]:
    """Per code of the 60/30/10 mix: its symbols (frames, S) and noise
    variances, each frame within spread_db of its code's waterfall."""
    gen = _generator(seed)
    counts = {"A": 0, "B": int(0.3 * case["frames"]), "C": int(0.1 * case["frames"])}
    counts["A"] = case["frames"] - counts["B"] - counts["C"]
    out = []
    for name, frames in counts.items():
        c = _constellation("qam", workloads.MIXED_ORDERS[name])
        _, _, m, N, n = _edges(name)
        words = _codewords(name, frames, gen)
        ebn0 = workloads.WATERFALL_DB[name] + case["spread_db"] * (
            2.0 * torch.rand(frames, device="cuda", generator=gen, dtype=torch.float64) - 1.0)  # fmt: skip
        nv = 10.0 ** (-ebn0 / 10.0) / ((N - m) / n * c.bits_per_symbol)
        out.append((name, c, _awgn(_map(words, c), nv.float()[:, None], gen), nv.cpu().numpy()))
    return out


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    if kind == "llr":
        return _prepare_llr(case, seed)
    if kind == "decode":
        return dict(llrs=_binary_llrs(case, seed), code=_code(case["code"]), method=_method(case))
    if kind == "encode":
        code = _code(case["code"])
        _, _, m, N, _ = _edges(case["code"])
        bits = torch.randint(0, 2, (case["frames"], N - m), device="cuda", generator=_generator(seed), dtype=torch.int8)
        return dict(bits=bits, code=code)
    if kind == "mixed":
        # The receiver's buffers, workspace and captured graph.
        inputs = _mixed_inputs(case, seed)
        slots = [pipeline.CodeSlot(_code(n), c, x.shape[0], ck.MinSum(max_iterations=50)) for n, c, x, _ in inputs]
        receiver = pipeline.MixedReceiver(slots)
        receiver.load([x for _, _, x, _ in inputs], [nv for _, _, _, nv in inputs])
        receiver.capture()
        return dict(receiver=receiver)
    _, _, m, N, n = _edges(case["code"])
    c = _constellation("qam", case["order"])
    esn0_db = case["ebn0_db"] + 10.0 * math.log10((N - m) / n * c.bits_per_symbol)
    return dict(code=_code(case["code"]), constellation=c, esn0_db=[esn0_db], blocks=case["blocks"], rng=seed)


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------


def run(state: dict):
    if "symbols" in state:
        return ck.compute_llr(state["symbols"], noise_var=state["noise_var"], constellation=state["constellation"],
                              method=state["method"])  # fmt: skip
    if "llrs" in state:
        r = ck.decode(state["llrs"], code=state["code"], method=state["method"])
        return r.bits, r.llrs, r.valid, r.iterations
    if "bits" in state:
        return ck.encode(state["bits"], code=state["code"])
    if "receiver" in state:
        receiver = state["receiver"]
        receiver.run()
        return [(r.bits, r.llrs, r.valid, r.iterations) for r in receiver.results()]
    curve = ck.error_rate_curve(state["code"], constellation=state["constellation"], esn0_db=state["esn0_db"],
                                min_block_errors=state["blocks"], max_blocks=state["blocks"], rng=state["rng"])  # fmt: skip
    return {f: getattr(curve, f) for f in ("num_blocks", "bit_errors", "block_errors", "pre_fec_bit_errors",
                                           "detected_failures", "undetected_errors", "total_iterations")}  # fmt: skip


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------

# Operations of one message of one iteration: subtract, compare with the two
# smallest magnitudes, add (min-sum); two evaluations of phi, each a tanh and
# a log, and three additions (sum-product).
_EDGE_OPS = {"min_sum": 4, "sum_product": 7}


def _decode_work(name: str, frames: int, rule: str) -> tuple[float, float]:
    """LLRs read, posteriors, bits, counts and flags written; one iteration
    (every noisy frame needs at least one)."""
    checks, _, m, N, n = _edges(name)
    return frames * (8.0 * n + (N - m) + 5.0), frames * float(checks.size) * _EDGE_OPS[rule]


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "llr":
        c = _constellation(case["family"], case["order"])
        k, n = c.bits_per_symbol, case["symbols"]
        square = case["family"] == "qam" and k % 2 == 0
        metrics = 2 * (1 << (k // 2)) if square else c.order
        per_metric = (3 if square else 6) + (2 if case["method"] == "exact" else 1)
        return {"bytes": n * (8.0 + 4.0 * k), "flops": float(n) * metrics * per_metric}
    if kind == "decode":
        b, f = _decode_work(case["code"], case["frames"], case["rule"])
        return {"bytes": b, "flops": f}
    if kind == "encode":
        checks, _, m, N, n = _edges(case["code"])
        return {"bytes": case["frames"] * float(N - m + n), "flops": case["frames"] * float(checks.size)}
    if kind == "mixed":
        counts = {"B": int(0.3 * case["frames"]), "C": int(0.1 * case["frames"])}
        counts["A"] = case["frames"] - counts["B"] - counts["C"]
        b = f = 0.0
        for name, frames in counts.items():
            n = _edges(name)[4]
            db, df = _decode_work(name, frames, "min_sum")
            k = int(math.log2(workloads.MIXED_ORDERS[name]))
            b, f = b + db - frames * n * (4.0 - 8.0 / k), f + df
        return {"bytes": b, "flops": f}
    # The blocks never leave the device: only the counters are output.
    b, f = _decode_work(case["code"], case["blocks"], "min_sum")
    return {"bytes": 56.0, "flops": f}


# ---------------------------------------------------------------------------
# 64-bit values
# ---------------------------------------------------------------------------


def _llr64(x: torch.Tensor, c: ck.Constellation, noise_var, method: str) -> torch.Tensor:
    """(..., S) symbols to (..., S k) LLRs from every point's metric in
    float64, noise_var broadcasting against the symbols."""
    x = x.to(torch.complex128)
    nv = torch.as_tensor(noise_var, dtype=torch.float64, device="cuda").expand(x.shape).reshape(-1)
    flat = x.reshape(-1)
    points = torch.from_numpy(np.asarray(c.points, np.complex64).astype(np.complex128)).cuda()
    ones = torch.from_numpy(np.asarray(c.bit_labels)).cuda() != 0
    out = torch.empty((flat.numel(), c.bits_per_symbol), dtype=torch.float64, device="cuda")
    step = max(1, (1 << 26) // c.order)
    for i in range(0, flat.numel(), step):
        d = torch.view_as_real(flat[i : i + step, None] - points)
        metric = -d.square().sum(-1) / nv[i : i + step, None]
        for b in range(c.bits_per_symbol):
            halves = metric[:, ~ones[:, b]], metric[:, ones[:, b]]
            if method == "maxlog":
                out[i : i + step, b] = halves[0].amax(1) - halves[1].amax(1)
            else:
                out[i : i + step, b] = halves[0].logsumexp(1) - halves[1].logsumexp(1)
    return out.reshape(*x.shape[:-1], -1)


@functools.lru_cache(maxsize=None)
def _layers(name: str) -> list[torch.Tensor]:
    """Per layer its rows' columns (rows, degree), the one after the last
    variable as filler: each check, in order, goes to the first layer none
    of whose checks shares a variable with it."""
    checks, variables, m, N, _ = _edges(name)
    order = np.lexsort((variables, checks))
    starts = np.searchsorted(checks[order], np.arange(m + 1))
    columns = variables[order].tolist()
    used, layers = [0] * N, []
    for i in range(m):
        row = columns[starts[i] : starts[i + 1]]
        taken = 0
        for v in row:
            taken |= used[v]
        at = (~taken & (taken + 1)).bit_length() - 1
        for v in row:
            used[v] |= 1 << at
        if at == len(layers):
            layers.append([])
        layers[at].append(row)
    width = max(len(r) for rows in layers for r in rows)
    return [torch.tensor([r + [N] * (width - len(r)) for r in rows], device="cuda") for rows in layers]


def _decode64(llrs: torch.Tensor, name: str, rule: str, iterations: int) -> torch.Tensor | None:
    """(frames, sent bits) LLRs to float64 posteriors: the layered recursion
    (min-sum with scale 0.875, or sum-product), each frame until its checks
    hold or the iterations are spent.  None when more than a hundredth of the
    frames end with checks that do not hold: such a frame wanders, and its
    last posterior is decided by rounding."""
    layers = _layers(name)
    N, n = _edges(name)[3:5]
    frames = llrs.shape[0]
    post = torch.zeros((frames, N + 1), dtype=torch.float64, device="cuda")
    post[:, :n] = llrs.reshape(frames, n).double()
    messages = [torch.zeros((frames, *c.shape), dtype=torch.float64, device="cuda") for c in layers]

    def phi(x):
        return -torch.log(torch.tanh(x.clamp(1e-7, 30.0) / 2.0))

    def unsolved(p):
        bad = torch.zeros(p.shape[0], dtype=torch.bool, device="cuda")
        for c in layers:
            bad |= ((p[:, c] < 0).sum(-1) % 2 != 0).any(1)
        return bad

    active = torch.nonzero(unsolved(post)).flatten()
    for _ in range(iterations):
        if not active.numel():
            break
        p = post[active]
        for c, store in zip(layers, messages, strict=True):
            edge = c < N
            q = p[:, c] - store[active]
            sign = torch.where(q < 0, -1.0, 1.0) * edge + (~edge)
            if rule == "min_sum":
                mag = q.abs().masked_fill(~edge, math.inf)
                low = mag.topk(2, dim=-1, largest=False).values
                first = torch.zeros_like(mag, dtype=torch.bool).scatter_(-1, mag.argmin(-1, keepdim=True), True)
                new = 0.875 * torch.where(first, low[..., 1:], low[..., :1])
            else:
                f = phi(q.abs()) * edge
                new = phi(f.sum(-1, keepdim=True) - f)
            new = new * sign * sign.prod(-1, keepdim=True)
            p[:, c.flatten()] = (q + new).flatten(1)
            p[:, N] = 0.0
            store[active] = new * edge
        post[active] = p
        active = active[unsolved(p)]
    return None if 100 * active.numel() > frames else post[:, :n]


def exact(case: dict, seed: int):
    """The float64 values of what :func:`run` returns; hard decisions, flags
    and counts are whole numbers."""
    kind = case["kind"]
    if kind == "llr":
        s = _prepare_llr(case, seed)
        return _llr64(s["symbols"], s["constellation"], s["noise_var"], s["method"])
    if kind == "decode":
        post = _decode64(_binary_llrs(case, seed), case["code"], case["rule"], case["iterations"])
        return None if post is None else (None, post, None, None)
    # A mixed step holds frames below their code's waterfall (see _decode64);
    # codewords and counts are whole numbers.
    return None
