"""What a user of this framework has it do, as cases that can be timed.

The model is the default one (``llmcp_b200.default_dims()``), random-init, as a Q8_0 container (llmcp-pack --quant
q8_0) or an unquantised one (--quant none).  A program loads it once and then serves prompts: ``prepare`` hands out the
loaded engine (or the AOT runtime) and a request's token ids, ``run`` serves that request from position 0.  Every
request clears the generation state first, so it can be repeated.

Kinds:
  request   Engine: a prompt, then single tokens, then perhaps a second prompt on top; logits to the host every time,
            as a sampling loop takes them.  The tokens are given (what a sampler would have drawn).
  generate  Engine: a prompt, greedy decoding on the device, and one step more with its logits.
  aot       the AOT ABI entries with host buffers (what llmcp-run and llmcp-benchmark call): prompt, then steps.
  batch     Engine with a batch of sequences: prompts one at a time, then all sequences decoded together, greedily on
            the device (exact arithmetic) or with their logits to the host at every step (fast arithmetic).
  score     Engine: the logits of every position of a text.
  linear    one Q8 projection on device pointers, input quantisation included (one row or many).
"""
import ctypes as C
import json

import numpy as np
import torch

import llmcp_b200 as L

ROOT = "model.language_model."
# Projections of the model: (rows, columns).
PROJECTIONS = [(9216, 2560), (8192, 2560), (4096, 2560), (1024, 2560), (2560, 4096), (2560, 9216)]
CAPACITIES = (256, 1160, 4608)  # positions an engine is created for: short chats, the benchmark's workload, long documents


def listed():
    return [
        # One projection of one token: the smallest call there is (benchmark: 9216 x 2560, one row).
        dict(name="linear_1_row", kind="linear", rows=1, n=9216, k=2560, fast=True),
        # The same projection over a prompt (benchmark: 1024 rows).
        dict(name="linear_1024_rows", kind="linear", rows=1024, n=9216, k=2560, fast=False),
        # The drop-in library's smallest call: one token into an empty cache, default (exact) arithmetic.
        dict(name="aot_first_token", kind="aot", prompt=1, steps=0, mode="exact", arena="q8_0"),
        # llmcp-run: a short question, then a sampling loop on the host.
        dict(name="aot_question", kind="aot", prompt=30, steps=40, mode="fast", arena="q8_0"),
        # A very short prompt: one ragged tile of rows.
        dict(name="prompt_23", kind="request", prompt=23, steps=0, second=0, mode="fast", arena="q8_0"),
        # The benchmark's prompt.
        dict(name="prompt_1024", kind="request", prompt=1024, steps=0, second=0, mode="fast", arena="q8_0"),
        # A prompt of odd length in the default arithmetic, bit for bit the reference's order.
        dict(name="prompt_517_exact", kind="request", prompt=517, steps=0, second=0, mode="exact", arena="q8_0"),
        # A long document, an answer, and a follow-up question on top of both.
        dict(name="document", kind="request", prompt=3001, steps=40, second=91, mode="fast", arena="q8_0"),
        # Greedy decoding that stays on the device, default arithmetic (benchmark: prompt, then 128 steps).
        dict(name="generate_exact", kind="generate", prompt=128, steps=128, mode="exact", arena="q8_0"),
        # Many sequences decoded together (benchmark: 64), short ones.
        dict(name="batch_64", kind="batch", batch=64, prompt=0, steps=12, mode="exact", arena="q8_0"),
        # Perplexity of a text: logits of every position.
        dict(name="score_160", kind="score", prompt=160, mode="fast", arena="q8_0"),
        # The unquantised arena (llmcp-pack's default): prompt and answer.
        dict(name="bf16_chat", kind="request", prompt=200, steps=32, second=0, mode="fast", arena="none"),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["linear", "linear", "request", "request", "generate", "aot", "batch", "score"])
    mode = rng.choice(["fast", "fast", "exact"])
    arena = "none" if rng.random() < 0.15 else "q8_0"
    if kind == "linear":
        n, k = rng.choice(PROJECTIONS)
        rows = 1 if rng.random() < 0.4 else _log(rng, 2, 2048)
        return dict(kind=kind, rows=rows, n=n, k=k, fast=rows == 1 and mode == "fast")  # many rows: one order of additions
    if kind == "request":
        prompt = _log(rng, 2, 2600 if mode == "fast" else 1000)
        second = _log(rng, 2, 150) if rng.random() < 0.4 else 0
        return dict(kind=kind, prompt=prompt, steps=rng.choice([0, rng.randint(1, 40)]), second=second, mode=mode, arena=arena)
    if kind == "generate":  # tokens are compared: the arithmetic whose results are fixed bit for bit
        return dict(kind=kind, prompt=_log(rng, 2, 700), steps=rng.randint(4, 100), mode="exact", arena="q8_0")
    if kind == "aot":
        return dict(kind=kind, prompt=_log(rng, 1, 700), steps=rng.randint(0, 40), mode=mode, arena="q8_0")
    if kind == "batch":
        batch = _log(rng, 2, 64)
        return dict(kind=kind, batch=batch, prompt=rng.choice([0, rng.randint(2, 120)]) if batch <= 8 else 0, steps=rng.randint(2, 6),
                    mode=mode, arena="q8_0")
    return dict(kind=kind, prompt=_log(rng, 2, 200), mode=mode, arena="q8_0")


# ---- the model ---------------------------------------------------------------------------------------------------

_containers, _engines, _runtimes = {}, {}, {}


def _layout(d, quantised):
    """Names, shapes and source types of the model's tensors, by group of layers (format: README, llmcp-pack)."""
    groups = []
    for g in range(d.layers // d.full_interval):
        tensors = []
        for i in range(d.full_interval):
            p = f"{ROOT}layers.{g * d.full_interval + i}."
            v = d.lin_v_heads * d.lin_v_dim
            tensors += [(p + "input_layernorm.weight", [d.hidden]), (p + "post_attention_layernorm.weight", [d.hidden])]
            if i < d.full_interval - 1:
                tensors += [(p + "linear_attn.in_proj_qkv.weight", [d.qkv_dim, d.hidden]),
                            (p + "linear_attn.in_proj_z.weight", [v, d.hidden]),
                            (p + "linear_attn.in_proj_a.weight", [d.lin_v_heads, d.hidden]),
                            (p + "linear_attn.in_proj_b.weight", [d.lin_v_heads, d.hidden]),
                            (p + "linear_attn.conv1d.weight", [d.qkv_dim, 1, d.conv_kernel]),
                            (p + "linear_attn.dt_bias", [d.lin_v_heads]), (p + "linear_attn.A_log", [d.lin_v_heads]),
                            (p + "linear_attn.norm.weight", [d.lin_v_dim]),
                            (p + "linear_attn.out_proj.weight", [d.hidden, v])]
            else:
                a = d.heads * d.head_dim
                tensors += [(p + "self_attn.q_proj.weight", [2 * a, d.hidden]),
                            (p + "self_attn.k_proj.weight", [d.kv_heads * d.head_dim, d.hidden]),
                            (p + "self_attn.v_proj.weight", [d.kv_heads * d.head_dim, d.hidden]),
                            (p + "self_attn.o_proj.weight", [d.hidden, a]),
                            (p + "self_attn.q_norm.weight", [d.head_dim]), (p + "self_attn.k_norm.weight", [d.head_dim])]
            tensors += [(p + "mlp.gate_proj.weight", [d.intermediate, d.hidden]), (p + "mlp.up_proj.weight", [d.intermediate, d.hidden]),
                        (p + "mlp.down_proj.weight", [d.hidden, d.intermediate])]
        groups.append(tensors)
    entries, cursor, stride = [], 64, 0

    def add(name, shape):
        nonlocal cursor
        dtype = "F32" if name.endswith(("A_log", "linear_attn.norm.weight")) else "BF16"
        size = int(np.prod(shape)) * (4 if dtype == "F32" else 2)
        source = size
        if quantised and len(shape) == 2:
            dtype, size = "Q8_0", shape[0] * (shape[1] // 32) * 34
        cursor = (cursor + 63) // 64 * 64
        entries.append(dict(name=name, shape=shape, dtype=dtype, offset=cursor, size=size, source_size=source))
        cursor += size

    add(ROOT + "embed_tokens.weight", [d.vocab, d.hidden])
    for tensors in groups:
        start = cursor
        for name, shape in tensors:
            add(name, shape)
        stride = (cursor - start + 63) // 64 * 64
        cursor = start + stride
    add(ROOT + "norm.weight", [d.hidden])
    total = (cursor + 63) // 64 * 64
    manifest = dict(alignment=64, group_stride=stride, header_bytes=64, model="random-init", num_groups=len(groups),
                    quantization="q8_0" if quantised else "none", tensors=entries, total_bytes=total)
    if quantised:
        manifest.update(block_size=32, quant_layout="q8_0_p4")
    return manifest


def _values(name, shape, generator):
    """Random-init values on the GPU: linears N(0, 0.02), norm gains around 1, decay rates and step sizes over the range
    such layers are initialised with.  The projections back into the residual stream are small beside the embeddings, as in a
    trained model, where a layer moves the stream a little: at equal size the forward is chaotic (it rounds to int8 some 230
    times, and two orders of addition then differ by 14 % of the logits' norm), and nothing could be compared."""
    def normal(std):
        return torch.randn(shape, generator=generator, device="cuda") * std
    if name.endswith("embed_tokens.weight"):
        return normal(1.0)
    if name.endswith(("out_proj.weight", "o_proj.weight", "down_proj.weight")):
        return normal(0.0006)
    if name.endswith("conv1d.weight"):
        return normal(0.5)
    if name.endswith("A_log"):
        return torch.log(1 + 15 * torch.rand(shape, generator=generator, device="cuda"))
    if name.endswith("dt_bias"):
        return normal(0.5) - 3.0
    if name.endswith("linear_attn.norm.weight"):
        return 1 + normal(0.1)
    if name.endswith(("norm.weight", "layernorm.weight")):  # stored zero-centred
        return normal(0.1)
    return normal(0.02)


def _q8_records(w):
    """Q8_0 blocks of 32 in the four-row lane layout: per (4 rows, block) 4 f16 scales, then 8 words x 4 rows x 4 bytes."""
    n, k = w.shape
    b = w.view(n, k // 32, 32)
    scale = b.abs().amax(-1, keepdim=True) / 127
    q = torch.clamp(torch.round(b / scale.clamp_min(1e-30)), -127, 127).to(torch.int8)
    record = torch.empty(n // 4, k // 32, 136, dtype=torch.uint8, device=w.device)
    record[:, :, :8] = scale.view(n // 4, 4, k // 32).permute(0, 2, 1).contiguous().to(torch.float16).view(torch.uint8).view(n // 4, k // 32, 8)
    record[:, :, 8:] = q.view(n // 4, 4, k // 32, 8, 4).permute(0, 2, 3, 1, 4).reshape(n // 4, k // 32, 128).view(torch.uint8)
    return record


def container(arena):
    """The packed model file in host memory, built once per process (what a program maps from disk)."""
    if arena not in _containers:
        manifest = _layout(L.default_dims(), arena == "q8_0")
        text = (json.dumps(manifest, separators=(",", ":"), sort_keys=True) + "\n").encode()
        total = manifest["total_bytes"]
        data = np.zeros(total + len(text), dtype=np.uint8)
        host = torch.from_numpy(data)
        generator = torch.Generator(device="cuda").manual_seed(7)
        for t in manifest["tensors"]:
            at, rows = t["offset"], t["shape"][0]
            step = 16384 if len(t["shape"]) == 2 else rows  # rows at a time: the f32 values never exist whole
            for r in range(0, rows, step):
                shape = [min(step, rows - r)] + t["shape"][1:]
                w = _values(t["name"], shape, generator)
                raw = _q8_records(w) if t["dtype"] == "Q8_0" else w.to(torch.bfloat16 if t["dtype"] == "BF16" else torch.float32)
                raw = raw.contiguous().view(torch.uint8).reshape(-1)
                host[at:at + raw.numel()].copy_(raw)
                at += raw.numel()
        data[total:] = np.frombuffer(text, dtype=np.uint8)
        header = b"LLMCPWGT" + b"".join(v.to_bytes(s, "little") for v, s in ((1, 4), (64, 4), (total, 8), (total, 8), (len(text), 8)))
        data[:len(header)] = np.frombuffer(header, dtype=np.uint8)
        del w, raw
        torch.cuda.empty_cache()
        _containers[arena] = data
    return _containers[arena]


def _capacity(positions):
    return next(c for c in CAPACITIES if c >= positions)


def _engine(arena, mode, capacity, batch=1):
    """The loaded engine: a program keeps it over its requests.  The one used last is kept here."""
    key = (arena, mode, capacity, batch)
    if key not in _engines:
        _engines.clear()
        _engines[key] = L.Engine(container(arena), capacity=capacity, mode=mode, batch=batch)
    return _engines[key]


def _runtime(mode, capacity):
    key = (mode, capacity)
    if key not in _runtimes:
        _runtimes.clear()
        L.lib().llmcp_b200_release_all()
        runtime, before = L.AotRuntime(), L.get_mode()
        if not runtime.init(max_sequence=capacity):
            raise RuntimeError("the AOT library did not load")
        arena = L.Arena().from_buffer(container("q8_0"))
        L.set_mode(mode)  # of the session that the first call opens
        try:
            runtime.forward(arena, [0], 0, 1)
        finally:
            L.set_mode(before)
        _runtimes[key] = runtime, arena
    return _runtimes[key]


# ---- cases -------------------------------------------------------------------------------------------------------


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng([seed, 1])
    if kind == "linear":
        return _prepare_linear(case, seed)
    vocab = L.default_dims().vocab
    state = dict(case=case)

    def tokens(*shape):
        return rng.integers(0, vocab, size=shape, dtype=np.int64)

    if kind == "request":
        positions = case["prompt"] + case["steps"] + case["second"]
        state.update(prompt=tokens(case["prompt"]), answer=tokens(case["steps"]), second=tokens(case["second"]),
                     engine=_engine(case["arena"], case["mode"], _capacity(positions)))
    elif kind == "generate":
        positions = case["prompt"] + case["steps"] + 1
        state.update(prompt=tokens(case["prompt"]), engine=_engine(case["arena"], case["mode"], _capacity(positions)))
    elif kind == "aot":
        runtime, arena = _runtime(case["mode"], _capacity(case["prompt"] + case["steps"]))
        state.update(prompt=tokens(case["prompt"]).tolist(), answer=tokens(case["steps"]).tolist(), runtime=runtime, arena=arena,
                     logits=[np.zeros(vocab, dtype=np.float32) for _ in range(case["steps"] + 1)])
    elif kind == "batch":
        positions = case["prompt"] + case["steps"] + 1
        state.update(prompts=tokens(case["batch"], case["prompt"]), answers=tokens(case["steps"] + 1, case["batch"]),
                     engine=_engine(case["arena"], case["mode"], _capacity(positions), case["batch"]))
    else:
        state.update(prompt=tokens(case["prompt"]), engine=_engine(case["arena"], case["mode"], _capacity(case["prompt"])))
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "linear":
        return _run_linear(state)
    if kind == "aot":
        runtime, arena, out = state["runtime"], state["arena"], state["logits"]
        at = len(state["prompt"])
        runtime.forward(arena, state["prompt"], 0, at, out[0])
        for i, token in enumerate(state["answer"]):
            runtime.forward(arena, [token], at + i, at + i + 1, out[i + 1])
        return out
    engine = state["engine"]
    engine.reset()
    if kind == "score":
        return engine.forward_all(state["prompt"], 0)
    if kind == "batch":
        for i, prompt in enumerate(state["prompts"]):
            if len(prompt):
                engine.select_sequence(i)
                engine.forward(prompt, 0, want_logits=False)
        if case["mode"] == "fast":  # a sampling loop on the host
            return [engine.decode_batch(tokens, case["prompt"] + i)[0] for i, tokens in enumerate(state["answers"])]
        tokens, _ = engine.generate_batch(state["answers"][0], case["prompt"], case["steps"])
        logits, _ = engine.decode_batch(tokens[-1], case["prompt"] + case["steps"])
        return tokens, logits
    logits, token = engine.forward(state["prompt"], 0)
    at = len(state["prompt"])
    if kind == "generate":
        tokens, _ = engine.generate(token, at, case["steps"])
        last, _ = engine.forward(tokens[-1:], at + case["steps"])
        return logits, tokens, last
    out = [logits]
    for i in range(case["steps"]):
        out.append(engine.forward(state["answer"][i:i + 1], at + i)[0])
    if case["second"]:
        out.append(engine.forward(state["second"], at + case["steps"])[0])
    return out


def _prepare_linear(case, seed):
    """Weights in the device layout (repacked once), the input rows in bf16, the buffers a caller keeps and the calls."""
    m, n, k = case["rows"], case["n"], case["k"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    lib, i, p, stream = L.lib(), C.c_int64, lambda t: C.c_void_p(t.data_ptr()), C.c_void_p(torch.cuda.current_stream().cuda_stream)

    def empty(dtype, *shape):
        return torch.empty(shape, dtype=dtype, device="cuda")

    x = torch.randn(m, k, generator=g, device="cuda").to(torch.bfloat16)
    records = _q8_records(torch.randn(n, k, generator=g, device="cuda") * 0.02)
    wq, wd, aq, scales = empty(torch.int8, n, k), empty(torch.float16, n, k // 32), empty(torch.int8, m, k), empty(torch.float32, m, k // 32)
    y, status = empty(torch.bfloat16, m, n), torch.zeros(1, dtype=torch.int32, device="cuda")
    _call(lib.llmcp_dev_repack_q8, p(records), i(n), i(k), p(wq), p(wd), stream)
    keep = [x, wq, wd, aq, scales, y, status]
    calls = [(lib.llmcp_dev_act_quant, p(x), 1, i(m), i(k), p(aq), p(scales), stream)]
    if m == 1:
        calls.append((lib.llmcp_dev_gemv_q8, p(aq), p(scales), i(k), p(wq), p(wd), i(n), p(y), 1, 0, 0, 3 | (16 if case["fast"] else 0), stream))
    else:
        pitch = lib.llmcp_dev_gemm_q8_tma_scale_pitch
        pitch.restype = C.c_int64
        ws, at = empty(torch.float32, k // 32, n), empty(torch.float32, k // 32, pitch(i(m)))
        keep += [ws, at]
        _call(lib.llmcp_dev_q8_gemm_planes, p(wq), p(wd), 1, i(n), i(k), None, p(ws), stream)
        calls += [(lib.llmcp_dev_q8_gemm_planes, p(aq), p(scales), 0, i(m), i(k), None, p(at), stream),
                  (lib.llmcp_dev_gemm_q8_tma, 1, p(aq), p(at), i(m), i(k), p(wq), p(ws), i(n), p(y), 1, 0, p(status), C.c_uint32(0), 0, stream)]
    torch.cuda.synchronize()
    return dict(case=case, calls=calls, keep=keep, y=y)


def _call(function, *arguments):
    if function(*arguments):
        raise L.LlmcpError(L.last_error())


def _run_linear(state):
    for call in state["calls"]:
        _call(*call)
    return state["y"]


# ---- what a pass cannot do without -------------------------------------------------------------------------------


def _forward_work(arena, rows, context, heads=1):
    """Bytes and flops of one forward over ``rows`` tokens behind ``context`` cached ones with ``heads`` rows of logits."""
    d = L.default_dims()
    v, a = d.lin_v_heads * d.lin_v_dim, d.heads * d.head_dim
    per_linear = (d.qkv_dim + v + 2 * d.lin_v_heads) * d.hidden + d.hidden * v
    per_full = (2 * a + 2 * d.kv_heads * d.head_dim) * d.hidden + d.hidden * a
    body = d.linear_layers * per_linear + d.full_layers * per_full + d.layers * 3 * d.intermediate * d.hidden
    weight = 2.0 if arena == "none" else 34 / 32
    state = d.linear_layers * d.lin_v_heads * d.lin_k_dim * d.lin_v_dim * 4 * 2
    keys = context + rows
    pairs = rows * context + rows * (rows + 1) / 2
    kv = d.full_layers * 2 * d.kv_heads * d.head_dim * 2
    return dict(weights=(body + d.vocab * d.hidden) * weight, other=state + keys * kv + rows * kv + heads * d.vocab * 4,
                flops=2 * rows * body + 2 * heads * d.vocab * d.hidden + d.full_layers * 4 * pairs * a
                + d.linear_layers * rows * d.lin_v_heads * 7 * d.lin_k_dim * d.lin_v_dim)


def work(case):
    kind = case["kind"]
    if kind == "linear":
        m, n, k = case["rows"], case["n"], case["k"]
        return dict(bytes=n * k * 34 / 32 + m * k * 2 + m * n * 2, flops=2 * m * n * k)
    calls = []  # (rows, context, rows of logits, sequences)
    prompt, steps = case["prompt"], case.get("steps", 0)
    if kind == "score":
        calls.append((prompt, 0, prompt, 1))
    elif kind == "batch":
        calls += [(prompt, 0, 1, 1)] * (case["batch"] if prompt else 0)
        calls += [(1, prompt + i, 1, case["batch"]) for i in range(steps + 1)]
    else:
        calls.append((prompt, 0, 1, 1))
        calls += [(1, prompt + i, 1, 1) for i in range(steps + (kind == "generate"))]
        if case.get("second"):
            calls.append((case["second"], prompt + steps, 1, 1))
    total = dict(bytes=0.0, flops=0.0)
    for rows, context, heads, sequences in calls:
        w = _forward_work(case["arena"], rows, context, heads)
        total["bytes"] += w["weights"] + sequences * w["other"]
        total["flops"] += sequences * w["flops"]
    return total


def tolerance(case):
    """Exact arithmetic: every bit.  Fast arithmetic, one projection: an f32 sum in another order moves a bf16 rounding here
    and there (one step of 2^-8 of a value).  Fast arithmetic, the model: another order of the f32 sums (the exact mode's)
    moved the logits by 0.0123 to 0.0131 of their norm, whatever the call, 0.0075 with bf16 weights, where the order is not
    fixed in either mode."""
    if case["kind"] == "linear":
        return {"rel": 1e-3, "max": 2.0 ** -7} if case["fast"] else "exact"
    return {"rel": 0.03} if case["mode"] == "fast" or case["arena"] == "none" else "exact"
