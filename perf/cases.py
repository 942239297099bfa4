"""What a user of the engine has it do, as cases that can be timed and checked.

Every case is a batch of sequences served by ``LLMEngine.feed`` with tokens that are given in advance (replaying a trace, scoring text):
the scheduler, the cache, the CUDA graphs of decode steps, the eager prompt steps and all kernels are those of ``generate`` and of the
server, but the outputs are logits that can be compared.  One pass opens the sequences as they arrive, feeds each prompt in portions of at
most ``BATCH`` tokens a step beside the sequences that already decode, then ``steps`` tokens one by one, and closes them.  The results are
the logits at the end of each prompt (the first token's) and of the last token; a caller of every other step would read ids only.

bf16 weights at random, of the shapes that the package's presets name; random token ids.
"""
import math

import torch

from jittorinfer_b200.models import registry, weights as deepseek_weights
from jittorinfer_b200.models.deepseek2 import DeepSeek2Model
from jittorinfer_b200.runtime.engine import EngineConfig, LLMEngine

BATCH = 2048                     # tokens of one step (the engine's default)
BUCKETS = (1, 2, 4, 8, 16, 32, 64)
SEED_STEP = 7919                 # weights and tokens come from different streams of one seed


# ---- the cases -----------------------------------------------------------------------------------------------------------------------
def _case(name, model, layers, seqs, prompt, steps, ragged=False, gap=0):
    return dict(name=name, model=model, layers=layers, seqs=seqs, prompt=prompt, steps=steps, ragged=ragged, gap=gap)


def listed():
    return [
        # one user: a prompt of a few tokens and an answer, the latency of a single decode step (headline workload at concurrency 1)
        _case("lite_chat_1", "lite", 27, 1, 5, 32),
        # the headline: eight requests with prompts of 1024 tokens each, decoded together
        _case("lite_chat_8", "lite", 27, 8, 1024, 32),
        # a full server: 64 short conversations of different lengths, decode dominates
        _case("lite_chat_64", "lite", 27, 64, 150, 32, ragged=True),
        # a whole prompt portion: scoring a text, the largest single step
        _case("lite_prompt_2048", "lite", 27, 1, 2048, 0),
        # time to first token of a short question, odd length, no graph
        _case("lite_prompt_77", "lite", 27, 1, 77, 0),
        # a long document in six portions and a short answer about it
        _case("lite_document", "lite", 27, 1, 12001, 16),
        # continuous batching: requests arrive every third step while the earlier ones decode
        _case("lite_arrivals", "lite", 27, 6, 700, 20, ragged=True, gap=3),
        # layer sizes of DeepSeek-V2 (low-rank queries, 128 heads, 160 experts in groups), four layers of it
        _case("v2_chat_8", "v2", 4, 8, 333, 16, ragged=True),
        # the folder architectures, whole: ragged prompts and answers of four users
        _case("nibalix_chat_4", "nibalix-lite", 12, 4, 777, 16, ragged=True),
        _case("lugovik_chat_4", "lugovik-lite", 12, 4, 777, 16, ragged=True),
        _case("zomavik_chat_4", "zomavik-lite", 10, 4, 777, 16, ragged=True),
        _case("rupatar_chat_4", "rupatar-lite", 12, 4, 777, 16, ragged=True),
    ]


def draw(rng):
    """Sequences, prompt lengths, answers and arrivals of the listed ranges; every second case is the plain model."""
    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    full = {c["model"]: c["layers"] for c in listed()}
    most = max(_cost(c) for c in listed())
    while True:
        model = "lite" if rng.random() < 0.5 else rng.choice(sorted(full))
        seqs = spread(1, 64) if model == "lite" else spread(1, 16)
        prompt = spread(3, 12000 if model == "lite" else 3000)
        steps = 0 if rng.random() < 0.25 else rng.randint(8, 32)
        gap = rng.choice([0, 0, 1, 3]) if seqs <= 24 else 0
        case = _case("", model, full[model], seqs, prompt, steps, ragged=rng.random() < 0.5, gap=gap)
        del case["name"]
        if seqs * (prompt + steps) <= 12288 and _cost(case) <= most:
            return case


def _hparams(case):
    hp = registry.preset(case["model"])
    if hasattr(hp, "replace"):
        return hp.replace(n_layer=case["layers"])
    if case["layers"] != hp.n_layer:
        raise ValueError("the folder architectures are taken whole")
    return hp


def _lengths(case):
    """Prompt lengths: all equal, or spread evenly from ``prompt`` down to a quarter of it."""
    p, n = case["prompt"], case["seqs"]
    return [max(1, p - 3 * p * i // (4 * n)) if case["ragged"] else p for i in range(n)]


def _schedule(case):
    """Per step the list of (sequence, first token, tokens, places among them whose logits are wanted)."""
    lens, steps = _lengths(case), case["steps"]
    at, out, now = [0] * len(lens), [], 0
    while any(a < n + steps for a, n in zip(at, lens)):
        step, room = [], BATCH
        live = [i for i in range(len(lens)) if i * case["gap"] <= now and at[i] < lens[i] + steps]
        for i in [i for i in live if at[i] >= lens[i]] + [i for i in live if at[i] < lens[i]]:      # decoding ones first
            n = 1 if at[i] >= lens[i] else min(lens[i] - at[i], room)
            if n == 0:
                continue
            end = at[i] + n
            step.append((i, at[i], n, [n - 1] if end in (lens[i], lens[i] + steps) else []))
            at[i], room = end, room - n
        if step:
            out.append(step)
        now += 1
    return out


# ---- inputs, pass ----------------------------------------------------------------------------------------------------------------------
def _weights(hp, seed, device="cuda"):
    """(name, tensor) pairs as a checkpoint would give them, drawn on the GPU.  Of trained stacks they keep that no sublayer outweighs the
    residual stream: embedding rows have elements around one, output projections are smaller by the root of twice the layers, those of
    routed experts by their number as well (with plain random matrices a near tie between two experts would decide most of the logits)."""
    arch = registry.for_hparams(hp)
    if arch.iter_random is None:
        pairs = deepseek_weights.iter_random(hp, seed=seed, dtype=torch.bfloat16, device=device, fast=True)
    else:
        pairs = arch.iter_random(hp, seed=seed, dtype=torch.bfloat16, device=device)
    for name, t in pairs:
        if name == "token_embd.weight":
            t *= 50
        elif name.endswith((".o", ".down", "attn_output.weight", "ffn_down.weight", "ffn_down_exps.weight", "ffn_down_shexp.weight")):
            t *= (2 * hp.n_layer) ** -0.5
        if name.endswith("ffn_down_exps.weight") or ".mlp.e" in name and name.endswith(".down"):
            t *= 1 / 6                                   # six experts a token in every shape taken here
        yield name, t


def _tokens(case, hp, seed):
    gen = torch.Generator().manual_seed(seed * SEED_STEP + 1)
    return [torch.randint(0, hp.n_vocab, (n + case["steps"],), generator=gen) for n in _lengths(case)]


def prepare(case, seed):
    hp = _hparams(case)
    arch = registry.for_hparams(hp)
    slot = (case["prompt"] + case["steps"] + 63) // 64 * 64
    model = (DeepSeek2Model if arch.load_config is None else arch.model)(hp, _weights(hp, seed), dtype=torch.bfloat16, device="cuda",
                                                                         max_positions=slot)
    top = next(b for b in BUCKETS if b >= case["seqs"])
    engine = LLMEngine(model, EngineConfig(n_ctx=slot * case["seqs"], n_batch=BATCH, n_parallel=case["seqs"], n_ctx_slot=slot,
                                           graph_buckets=tuple(b for b in BUCKETS if b <= top)))
    if case["steps"]:
        engine.warmup(("logits",))
    toks, lens = [t.tolist() for t in _tokens(case, hp, seed)], _lengths(case)
    plan = []
    for step in _schedule(case):
        entries = [(i, toks[i][a:a + n], want) for i, a, n, want in step]
        plan.append((entries, [i for i, a, n, _ in step if a + n == lens[i] + case["steps"]]))
    return {"engine": engine, "plan": plan}


def run(state):
    engine, out = state["engine"], []
    for entries, finished in state["plan"]:
        logits = engine.feed(entries)
        if logits.shape[0]:
            out.append(logits)
        for key in finished:
            engine.end_feed(key)
    return out


# ---- what a pass cannot do without -----------------------------------------------------------------------------------------------------
def _shapes(hp):
    arch = registry.for_hparams(hp)
    if arch.load_config is None:
        return deepseek_weights.tensor_table(hp)
    import sys
    module = sys.modules[arch.model.__module__]
    return {k: tuple(128 if n is None else n for n in s) for k, s in module.tensor_table(hp).items()}


def _attention_layers(hp):
    """(window, bytes of a cached token, flops of a query on one key, bytes of a sequence's recurrent state) of every layer run."""
    if hasattr(hp, "kv_lora_rank"):
        return [(0, 2 * hp.kv_row, 2 * hp.n_head * (hp.qk_head_dim + hp.v_head_dim), 0)] * hp.n_layer
    out = []
    for i in getattr(hp, "runs", range(hp.n_layer)):
        m = hp.layers[i].mixer
        a = getattr(m, "left", m)                       # attention beside a recurrence, or the mixer itself
        r = getattr(m, "right", None if hasattr(a, "kv_rank") or hasattr(a, "kv_heads") and hasattr(a, "rot") else m)
        win, row, per_key, state = 0, 0, 0, 0
        if hasattr(a, "kv_rank"):
            win, row, per_key = a.window, 2 * a.kv_row, 2 * a.heads * (a.dim + a.rot_dim + a.vdim)
        elif hasattr(a, "rot"):
            win = getattr(a, "window", 0) or getattr(a, "chunk", 0)
            row, per_key = 2 * a.kv_heads * (a.dim + a.vdim), 2 * a.heads * (a.dim + a.vdim)
        if r is not None:
            if hasattr(r, "inner") and hasattr(r, "dt_rank"):
                state = 4 * r.inner * r.state
            elif hasattr(r, "width"):
                state = 4 * r.width
            else:
                state = 4 * r.heads * r.vdim * getattr(r, "dim", getattr(r, "state", 0))
        out.append((win, row, per_key, state))
    return out


def work(case):
    """Per step: every weight that its tokens use read once (of the experts as many as are hit on average), every cached row that they
    see read once per sequence, recurrent states read and written, logits written; two operations per weight and token."""
    hp, vocab_rows = _hparams(case), 0
    runs = list(getattr(hp, "runs", range(hp.n_layer)))
    dense, expert, n_experts, top, dim, head = 0, 0, {}, {}, 0, 0
    for name, shape in _shapes(hp).items():
        n = math.prod(shape)
        layer = int(name.split(".")[1]) if name.startswith("blk.") else int(name[1:name.index(".")]) if name[0] == "l" and name[1].isdigit() else -1
        times = runs.count(layer) if layer >= 0 else 1
        if name in ("embed", "token_embd.weight"):
            dim = shape[1]
        elif name in ("head", "output.weight"):
            head = n
        elif "_exps." in name or ".mlp.e" in name:
            expert += n * times
            m = hp if hasattr(hp, "n_expert") else hp.layers[layer].mlp
            n_experts, top = getattr(m, "n_expert", getattr(m, "experts", 0)), getattr(m, "n_expert_used", getattr(m, "top", 0))
        else:
            dense += n * times
    layers = _attention_layers(hp)
    nbytes = flops = 0.0
    for step in _schedule(case):
        t = sum(n for _, _, n, _ in step)
        rows = len(step) if t == len(step) else sum(len(w) for *_, w in step)        # a decode step has every sequence's next token
        nbytes += 2 * (dense + t * dim) + (2 * head + 4 * rows * hp.n_vocab if rows else 0)
        flops += 2.0 * (dense * t + head * rows)
        if expert:
            nbytes += 2 * expert * (1 - (1 - top / n_experts) ** t)
            flops += 2.0 * expert * top / n_experts * t
        for win, row, per_key, state in layers:
            for _, a, n, _ in step:
                nbytes += 2 * state + row * (min(a + n, win + n - 1) if win else a + n)
                flops += per_key * sum(min(p + 1, win) if win else p + 1 for p in range(a, a + n))
    return {"bytes": nbytes, "flops": flops}


def _cost(case):
    w = work(case)
    return max(w["bytes"] / 6e12, w["flops"] / 1.4e15)


def tolerance(case):
    """bf16 activations through many layers: four times the distance from ``exact`` that was measured.  Of single tokens some are further
    off, where a near tie between experts falls the other way; most so with scores scaled by 16 (v2)."""
    return {"rel": {"lite": 0.05, "v2": 0.12, "nibalix-lite": 0.008, "lugovik-lite": 0.07, "zomavik-lite": 0.03, "rupatar-lite": 0.03}[case["model"]]}


# ---- the same in 64 bits ---------------------------------------------------------------------------------------------------------------
# Sequences side by side [B, n, ...], shorter ones filled up at the end (every mechanism looks backwards only).
def _mm(x, w):
    return x @ w.double().T


def _silu(x):
    return x * torch.sigmoid(x)


def _softplus(x):
    return torch.log1p(torch.exp(-x.abs())) + x.clamp_min(0)


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _angles(n, freqs, device):
    return torch.arange(n, dtype=torch.float64, device=device)[:, None] * torch.tensor(freqs, dtype=torch.float64, device=device)


def _yarn(dims, base, factor, original, fast, slow):
    at = lambda turns: dims * math.log(original / (2 * math.pi * turns)) / (2 * math.log(base))      # noqa: E731
    lo, hi = max(math.floor(at(fast)), 0), min(math.ceil(at(slow)), dims - 1)
    out = []
    for i in range(dims // 2):
        f, ramp = base ** (-2.0 * i / dims), min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0)
        out.append(f / factor * ramp + f * (1 - ramp))
    return out


def _rotate(v, freqs, neighbours, mult=1.0):
    """v [B, n, heads, D]: pairs (2i, 2i + 1) or (i, i + half) of the first 2 * len(freqs) elements turn."""
    half, a = len(freqs), _angles(v.shape[1], freqs, v.device)
    c, s = (torch.cos(a) * mult)[:, None], (torch.sin(a) * mult)[:, None]
    i0, i1 = (slice(0, 2 * half, 2), slice(1, 2 * half, 2)) if neighbours else (slice(0, half), slice(half, 2 * half))
    out = v.clone()
    out[..., i0], out[..., i1] = v[..., i0] * c - v[..., i1] * s, v[..., i0] * s + v[..., i1] * c
    return out


def _attend(q, k, v, scale, sees, denominator=None, softcap=0.0, shift=True):
    """q [B, n, H, D], k [B, m, G, D], v [B, m, G, V], ``sees(query positions [r, 1], key indices [1, m])``; ``denominator`` [H]: logits of
    a key without a value."""
    B, n, H, _ = q.shape
    G = k.shape[2]
    out = torch.empty(B, n, H, v.shape[3], dtype=q.dtype, device=q.device)
    js = torch.arange(k.shape[1], device=q.device)[None]
    kt, vt = k.permute(0, 2, 3, 1).repeat_interleave(H // G, 1), v.transpose(1, 2).repeat_interleave(H // G, 1)
    rows = max(1, min(n, (1 << 28) // max(1, B * H * k.shape[1])))
    for r in range(0, n, rows):
        s = (q[:, r:r + rows].transpose(1, 2) @ kt) * scale
        if softcap:
            s = softcap * torch.tanh(s / softcap)
        s = s.masked_fill(~sees(torch.arange(r, min(n, r + rows), device=q.device)[:, None], js), -math.inf)
        top = s.max(-1, keepdim=True).values
        if denominator is not None:
            top = torch.maximum(top, denominator.view(1, H, 1, 1))
        e = torch.exp(s - top)
        total = e.sum(-1, keepdim=True)
        if denominator is not None:
            total = total + torch.exp(denominator.view(1, H, 1, 1) - top)
        out[:, r:r + rows] = ((e @ vt) / total).transpose(1, 2)
    return out.flatten(2)


def _causal(window=0, chunk=0):
    def sees(i, j):
        ok = j <= i
        if window:
            ok = ok & (i - j < window)
        if chunk:
            ok = ok & (j >= i // chunk * chunk)
        return ok
    return sees


def _short_conv(x, taps_w, bias=None):
    """x [B, n, ch], taps_w [ch, taps]: the last column meets the current row."""
    taps, n = taps_w.shape[1], x.shape[1]
    pad = torch.nn.functional.pad(x, (0, 0, taps - 1, 0))
    out = sum(taps_w[:, j].double() * pad[:, j:j + n] for j in range(taps))
    return out if bias is None else out + bias.double()


def _experts(h, ids, wts, ffn, n):
    """Sum over the chosen experts; ``ffn(e, rows, weights [rows, 1])`` is one expert's part."""
    x, flat, w = h.flatten(0, -2), ids.flatten(0, -2), wts.flatten(0, -2)
    out = torch.zeros_like(x)
    for e in range(n):
        t, k = torch.nonzero(flat == e, as_tuple=True)
        if t.numel():
            out[t] += ffn(e, x[t], w[t, k][:, None])
    return out.view_as(h)


def _gated(w, p, act=_silu):
    return lambda x: _mm(act(_mm(x, w[p + "gate"])) * _mm(x, w[p + "up"]), w[p + "down"])


def _deepseek(hp, w, tokens):
    """Logits' last input [B, n, d]: latent attention expanded per head, group-limited top-k experts, softmax scores."""
    H, dn, dr, dv, r, eps = hp.n_head, hp.qk_nope_head_dim, hp.qk_rope_head_dim, hp.v_head_dim, hp.kv_lora_rank, hp.rms_eps
    B, n = tokens.shape
    norm = lambda x, k: _rms(x, eps) * w[k].double()                                                # noqa: E731
    freqs = _yarn(dr, hp.rope_freq_base, hp.rope_scaling_factor, hp.rope_orig_ctx, hp.yarn_beta_fast, hp.yarn_beta_slow)
    scale = (1 + hp.rope_yarn_log_mul * math.log(hp.rope_scaling_factor)) ** 2 / math.sqrt(dn + dr)
    x = w["token_embd.weight"][tokens].double()
    for i in range(hp.n_layer):
        p = f"blk.{i}."
        h = norm(x, p + "attn_norm.weight")
        if hp.q_lora_rank:
            q = _mm(norm(_mm(h, w[p + "attn_q_a.weight"]), p + "attn_q_a_norm.weight"), w[p + "attn_q_b.weight"])
        else:
            q = _mm(h, w[p + "attn_q.weight"])
        q = q.view(B, n, H, dn + dr)
        ckv = _mm(h, w[p + "attn_kv_a_mqa.weight"])
        kv = _mm(norm(ckv[..., :r], p + "attn_kv_a_norm.weight"), w[p + "attn_kv_b.weight"]).view(B, n, H, dn + dv)
        k_pe = _rotate(ckv[:, :, None, r:], freqs, True)
        q = torch.cat([q[..., :dn], _rotate(q[..., dn:], freqs, True)], -1)
        k = torch.cat([kv[..., :dn], k_pe.expand(B, n, H, dr)], -1)
        x = x + _mm(_attend(q, k, kv[..., dn:], scale, _causal()), w[p + "attn_output.weight"])
        g = norm(x, p + "ffn_norm.weight")
        part = lambda kind, e=None: w[p + f"ffn_{kind}.weight"] if e is None else w[p + f"ffn_{kind}_exps.weight"][e]      # noqa: B023,E731
        if i < hp.n_layer_dense_lead:
            x = x + _mm(_silu(_mm(g, part("gate"))) * _mm(g, part("up")), part("down"))
            continue
        probs = torch.softmax(_mm(g, part("gate_inp")), -1)
        sel = probs
        if hp.n_group > 1:
            best = sel.unflatten(-1, (hp.n_group, -1)).max(-1).values
            keep = torch.zeros_like(best, dtype=torch.bool).scatter_(-1, best.topk(hp.topk_group, -1).indices, True)
            sel = sel.masked_fill(~keep.repeat_interleave(hp.n_expert // hp.n_group, -1), -1.0)
        ids = sel.topk(hp.n_expert_used, -1).indices
        wts = probs.gather(-1, ids) * hp.expert_weights_scale
        ffn = lambda e, t, wt: wt * _mm(_silu(_mm(t, part("gate", e))) * _mm(t, part("up", e)), part("down", e))           # noqa: B023,E731
        y = _experts(g, ids, wts, ffn, hp.n_expert)
        x = x + y + _mm(_silu(_mm(g, part("gate_shexp"))) * _mm(g, part("up_shexp")), part("down_shexp"))
    return norm(x, "output_norm.weight")


def _nibalix(hp, w, tokens):
    """Parallel mixer and experts behind sigmoid gates; windowed latent attention or minGRU, an input convolution ahead of the mixer."""
    B, n = tokens.shape
    norm = lambda x, k: _rms(x, hp.eps) * (1 + w[k].double())                                       # noqa: E731
    x, rows = norm(w["embed"][tokens].double(), "embed.norm"), {}
    for i, L in enumerate(hp.layers):
        p, m = f"l{i}.", L.mixer
        h = norm(x, p + "norm1")
        hm = h + _short_conv(h, w[p + "canon1"])
        if hasattr(m, "kv_rank"):
            freqs = [m.rope_base ** (-2.0 * j / m.rot_dim) for j in range(m.rot_dim // 2)]
            src = i if m.kv_from is None else m.kv_from
            if src == i:
                y = _mm(hm, w[p + "mix.dkv"])
                rows[i] = (_rms(y[..., :m.kv_rank], hp.eps) * w[p + "mix.dkv.norm"].double(), _rotate(y[:, :, None, m.kv_rank:], freqs, False))
            c, kr = rows[src]
            q = _mm(hm, w[p + "mix.q"]).view(B, n, m.heads, m.dim + m.rot_dim)
            q = torch.cat([q[..., :m.dim], _rotate(q[..., m.dim:], freqs, False)], -1)
            k = torch.cat([_mm(c, w[p + "mix.uk"]).view(B, n, m.heads, m.dim), kr.expand(B, n, m.heads, m.rot_dim)], -1)
            y = _attend(q, k, _mm(c, w[p + "mix.uv"]).view(B, n, m.heads, m.vdim), m.scale, _causal(m.window))
        else:
            z = torch.sigmoid(_mm(hm, w[p + "mix.z"]) + w[p + "mix.z.b"].double())
            u = _mm(hm, w[p + "mix.x"]) + w[p + "mix.x.b"].double()
            cand, g = torch.where(u >= 0, u + 0.5, torch.sigmoid(u)), _mm(hm, w[p + "mix.g"])
            s, ys = torch.zeros_like(z[:, 0]), []
            for t in range(n):
                s = s + z[:, t] * (cand[:, t] - s)
                ys.append(s)
            y = torch.stack(ys, 1) * _silu(g)
        y = torch.sigmoid(_mm(h, w[p + "rg1"]) + w[p + "rg1.b"].double()) * _mm(y, w[p + "mix.o"])
        e = L.mlp
        v, ids = torch.topk(_mm(h, w[p + "mlp.router"]) + w[p + "mlp.router.b"].double(), e.top, -1)
        moe = _experts(h, ids, torch.softmax(v, -1), lambda j, t, wt: wt * _gated(w, f"{p}mlp.e{j}.")(t), e.experts)       # noqa: B023
        y = y + torch.sigmoid(_mm(h, w[p + "rg2"]) + w[p + "rg2.b"].double()) * moe
        x = x + hp.residual_mult * y
    return norm(x, "final.norm")


def _matrix_state(q, k, v, decay, beta=None):
    """S <- diag(decay) S, [u = beta (v - S^T k) for v,] S <- S + k u^T, o = S^T q; q, k, decay [B, n, H, K], v [B, n, H, V]."""
    B, n, H, K = q.shape
    s, out = torch.zeros(B, H, K, v.shape[3], dtype=q.dtype, device=q.device), []
    for t in range(n):
        s = decay[:, t, :, :, None] * s
        u = v[:, t]
        if beta is not None:
            u = beta[:, t, :, None] * (u - (k[:, t, :, None] @ s)[:, :, 0])
        s = s + k[:, t, :, :, None] * u[:, :, None]
        out.append((q[:, t, :, None] @ s)[:, :, 0])
    return torch.stack(out, 1)


def _lugovik_mixer(w, p, m, h, eps):
    B, n = h.shape[:2]
    lin = lambda k: _mm(h, w[p + k])                                                                # noqa: E731
    norm = lambda x, k: _rms(x, eps) * w[p + k].double()                                            # noqa: E731
    if hasattr(m, "groups"):                             # mamba2
        H, V, N, G, inner = m.heads, m.vdim, m.state, m.groups, m.heads * m.vdim
        z, xbc, dt = torch.split(lin("in"), [inner, inner + 2 * G * N, H], -1)
        x, b, c = torch.split(_silu(_short_conv(xbc, w[p + "conv"], w[p + "conv.b"])), [inner, G * N, G * N], -1)
        x = x.view(B, n, H, V)
        b, c = (y.view(B, n, G, N).repeat_interleave(H // G, 2) for y in (b, c))
        dt = _softplus(dt + w[p + "dt_bias"].double())
        decay = torch.exp(-torch.exp(w[p + "A_log"].double()) * dt)[..., None].expand(B, n, H, N)
        y = _matrix_state(c, b, dt[..., None] * x, decay) + w[p + "D"].double()[:, None] * x
        y = (y.flatten(2) * _silu(z)).unflatten(-1, (m.norm_groups, -1))
        return _mm(_rms(y, eps).flatten(2) * w[p + "norm"].double(), w[p + "o"])
    if hasattr(m, "kv_heads"):                           # channel_delta
        H, G, K, V = m.heads, m.kv_heads, m.dim, m.vdim
        unit = lambda x: x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)                       # noqa: E731
        q, k, v = (_silu(_short_conv(lin(c), w[p + c + ".conv"])) for c in "qkv")
        q, k = (unit(x.view(B, n, G, K)).repeat_interleave(H // G, 2) for x in (q, k))
        sp = _softplus(_mm(lin("a1"), w[p + "a2"]) + w[p + "dt_bias"].double()).view(B, n, H, K)
        decay = torch.exp(-torch.exp(w[p + "A_log"].double())[:, None] * sp)
        o = _matrix_state(q * K ** -0.5, k, v.view(B, n, H, V), decay, torch.sigmoid(lin("b")))
        o = norm(o, "norm") * torch.sigmoid(_mm(lin("g1"), w[p + "g2"])).view(B, n, H, V)
        return _mm(o.flatten(2), w[p + "o"])
    a, r = m.left, m.right                               # attention beside gated linear attention
    lin = lambda k, heads: _mm(h, w[p + k]).view(B, n, heads, -1)                                   # noqa: E731
    y = a.rot.yarn
    freqs, mult = _yarn(a.rot.dims, a.rot.base, y.factor, y.original, y.fast, y.slow), 0.1 * math.log(y.factor) + 1
    q, k = (_rotate(norm(lin("left." + c, g), f"left.{c}.norm"), freqs, False, mult) for c, g in (("q", a.heads), ("k", a.kv_heads)))
    zero = torch.zeros(a.heads, dtype=h.dtype, device=h.device)
    o = _attend(q, k, lin("left.v", a.kv_heads), a.scale, _causal(chunk=a.chunk), zero, a.softcap)
    o = (o.view(B, n, a.heads, -1) * torch.sigmoid(lin("left.g", a.heads))).flatten(2)
    left = _mm(o, w[p + "left.o"])
    z = _mm(_mm(h, w[p + "right.a1"]), w[p + "right.a2"]) + w[p + "right.a2.b"].double()
    alpha = torch.exp(-_softplus(-z) / r.tau).view(B, n, r.heads, r.dim)
    o = _matrix_state(lin("right.q", r.heads) * r.dim ** -0.5, lin("right.k", r.heads), lin("right.v", r.heads), alpha)
    right = _mm(norm(o, "right.norm").flatten(2) * _silu(_mm(h, w[p + "right.g"])), w[p + "right.o"])
    return m.left_scale * left + m.right_scale * right


def _lugovik(hp, w, tokens):
    norm = lambda x, k: _rms(x, hp.eps) * w[k].double()                                             # noqa: E731
    gelu = lambda x: torch.nn.functional.gelu(x, approximate="tanh")                                # noqa: E731
    x = w["embed"][tokens].double() * hp.embed_scale
    for i, L in enumerate(hp.layers):
        p = f"l{i}."
        x = x + norm(_lugovik_mixer(w, p + "mix.", L.mixer, norm(x, p + "norm1"), hp.eps), p + "norm1b")
        if L.ff is not None:
            x = x + norm(_gated(w, p + "mlp.", gelu)(norm(x, p + "norm2")), p + "norm2b")
    return norm(x, "final.norm")


def _zomavik_mixer(w, p, m, h):
    """Attention with learned sinks beside a selective scan."""
    B, n = h.shape[:2]
    a, r = m.left, m.right
    freqs = [a.rot.base ** (-2.0 * j / a.rot.dims) for j in range(a.rot.dims // 2)]
    q, k, v = ((_mm(h, w[f"{p}left.{c}"]) + w[f"{p}left.{c}.b"].double()).view(B, n, g, -1)
               for c, g in (("q", a.heads), ("k", a.kv_heads), ("v", a.kv_heads)))
    o = _attend(_rotate(q, freqs, False), _rotate(k, freqs, False), v, a.scale, _causal(), w[p + "left.sink"].double(), a.softcap)
    left = _mm(o, w[p + "left.o"])
    p += "right."
    x, z = torch.split(_mm(h, w[p + "in"]), r.inner, -1)
    x = _silu(_short_conv(x, w[p + "conv"], w[p + "conv.b"]))
    dt, b, c = torch.split(_mm(x, w[p + "x"]), [r.dt_rank, r.state, r.state], -1)
    dt = _softplus(_mm(dt, w[p + "dt"]) + w[p + "dt.b"].double())
    neg_a, s, ys = -torch.exp(w[p + "A_log"].double()), torch.zeros(B, r.inner, r.state, dtype=h.dtype, device=h.device), []
    for t in range(n):
        s = torch.exp(dt[:, t, :, None] * neg_a) * s + (dt[:, t] * x[:, t])[..., None] * b[:, t, None]
        ys.append((s @ c[:, t, :, None])[..., 0])
    y = (torch.stack(ys, 1) + w[p + "D"].double() * x) * _silu(z)
    return m.left_scale * left + m.right_scale * _mm(y, w[p + "o"])


def _zomavik(hp, w, tokens):
    norm = lambda x, k: _rms(x, hp.eps) * w[k].double()                                             # noqa: E731
    x = x0 = w["embed"][tokens].double() * hp.embed_scale
    starts = hp.passes
    for k, i in enumerate(hp.runs):
        if k in starts:
            x = _mm(torch.cat([x, x0], -1), w["loop.in"])
        p, m = f"l{i}.", hp.layers[i].mlp
        h = norm(x, p + "norm2")                         # both sublayers read the same row
        x = x + _zomavik_mixer(w, p + "mix.", hp.layers[i].mixer, norm(x, p + "norm1")) * w[p + "ls1"].double()
        probs = torch.softmax(_mm(h, w[p + "mlp.router"]), -1)
        v, ids = probs.topk(m.top, -1)                   # one group of experts in the shape taken here
        y = _experts(h, ids, v / v.sum(-1, keepdim=True), lambda e, t, wt: wt * _gated(w, f"{p}mlp.e{e}.")(t), m.experts)      # noqa: B023
        y = y + torch.sigmoid(_mm(h, w[p + "mlp.shared.sg"])) * _gated(w, p + "mlp.shared.")(h)
        x = x + y * w[p + "ls2"].double()
    return norm(x, "final.norm")


def _rupatar_mixer(w, p, m, h, eps, first):
    B, n = h.shape[:2]
    H = m.heads
    lin = lambda k, heads: _mm(h, w[p + k]).view(B, n, heads, -1)                                   # noqa: E731
    bias = lambda k: w[p + k + ".b"].double()                                                       # noqa: E731
    if hasattr(m, "gate_cap"):                           # mlstm
        q, k, v = (lin(c, H) for c in "qkv")
        gates = [m.gate_cap * torch.tanh((_mm(h, w[p + c]) + bias(c)) / m.gate_cap) for c in "if"]
        gi, gf = gates[0], -_softplus(-gates[1])
        s, nrm, top = (torch.zeros(B, H, *z, dtype=h.dtype, device=h.device) for z in ((m.dim, m.vdim), (m.dim,), ()))
        out = []
        for t in range(n):
            new = torch.maximum(gf[:, t] + top, gi[:, t])
            keep, put = torch.exp(gf[:, t] + top - new)[..., None], torch.exp(gi[:, t] - new)[..., None]
            s = keep[..., None] * s + (put * k[:, t])[..., None] * v[:, t, :, None]
            nrm, top = keep * nrm + put * k[:, t], new
            qt = q[:, t] * m.dim ** -0.5
            size = torch.maximum((nrm * qt).sum(-1).abs(), torch.exp(-top)) + 1e-6
            out.append((qt[:, :, None] @ s)[:, :, 0] / size[..., None])
        y = _rms(torch.stack(out, 1), eps).flatten(2) * w[p + "norm"].double() * torch.sigmoid(_mm(h, w[p + "g"]))
        return _mm(y, w[p + "o"])
    if not hasattr(m, "kv_heads"):                       # hgrn2
        low = w[p + "lower"].double()
        f = (low + (1 - low) * torch.sigmoid(_mm(h, w[p + "f"]) + bias("f"))).view(B, n, H, -1)
        o = _matrix_state(_silu(lin("q", H)), 1 - f, lin("v", H), f)
        return _mm((_rms(o, eps) * w[p + "norm"].double()).flatten(2), w[p + "o"])
    freqs = [m.rot.base ** (-2.0 * j / m.rot.dims) / m.rot.stretch for j in range(m.rot.dims // 2)]
    q, k, v = (lin(c, g) + bias(c).view(g, -1) for c, g in (("q", H), ("k", m.kv_heads), ("v", m.kv_heads)))
    q, k = (_rms(_rotate(x, freqs, True), eps) for x in (q, k))
    if m.v_mix:
        if first:
            lam = w[p + "vmix"].double()
            v = (1 - lam) * v + lam * first[0]
        else:
            first.append(v)
    size, pool, full = m.window, m.pool, n // m.pool if m.pool else 0
    mean = lambda x: x[:, :full * pool].unflatten(1, (full, pool)).mean(2)                          # noqa: E731
    if full:
        k, v = torch.cat([k, mean(k)], 1), torch.cat([v, mean(v)], 1)

    def sees(i, j):                                      # tokens of the window, blocks that end before it
        near = (j <= i) & (j < n)
        if size:
            near = near & (i - j < size)
        return near | ((j >= n) & ((j - n) * max(pool, 1) + pool - 1 <= i - size)) if full else near
    o = _attend(q, k, v, m.scale, sees, torch.zeros(H, dtype=h.dtype, device=h.device))
    return _mm(o * torch.sigmoid(_mm(h, w[p + "g"])), w[p + "o"]) + w[p + "o.b"].double()


def _rupatar(hp, w, tokens):
    norm = lambda x, k: _rms(x.unflatten(-1, (hp.groups, -1)), hp.eps).flatten(2) * w[k].double()   # noqa: E731
    gelu = torch.nn.functional.gelu
    x, first = w["embed"][tokens].double() * hp.embed_scale, []
    for i, L in enumerate(hp.layers):
        p, m = f"l{i}.", L.mlp
        x = x + _rupatar_mixer(w, p + "mix.", L.mixer, norm(x, p + "norm1"), hp.eps, first)
        h = norm(x, p + "norm2")
        one = lambda e, t: _mm(gelu(_mm(t, w[f"{p}mlp.{e}.up"])), w[f"{p}mlp.{e}.down"])            # noqa: B023,E731
        v, ids = torch.sigmoid(_mm(h, w[p + "mlp.router"])).topk(m.top, -1)
        x = x + _experts(h, ids, v, lambda e, t, wt: one(f"e{e}", wt * t), m.experts) + one("shared", h)      # noqa: B023
    return norm(x, "final.norm")


@torch.no_grad()
def exact(case, seed):
    hp, lens = _hparams(case), _lengths(case)
    w = dict(_weights(hp, seed))
    toks = _tokens(case, hp, seed)
    tokens = torch.zeros(len(toks), max(len(t) for t in toks), dtype=torch.int64)
    for i, t in enumerate(toks):
        tokens[i, :len(t)] = t
    arch = registry.for_hparams(hp).name
    rows = {"deepseek2": _deepseek, "Nibalix": _nibalix, "Lugovik": _lugovik, "Zomavik": _zomavik, "Rupatar": _rupatar}[arch](hp, w, tokens.cuda())
    head = w["output.weight" if arch == "deepseek2" else "head"]
    out = []
    for step in _schedule(case):
        at = [(i, a + k) for i, a, n, want in step for k in want]
        if at:
            y = _mm(rows[[i for i, _ in at], [p for _, p in at]], head)
            if arch == "Zomavik":
                y = hp.logit_softcap * torch.tanh(y * hp.logit_scale / hp.logit_softcap)
            out.append(y.cpu())
    return out
