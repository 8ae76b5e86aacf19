"""Fast mode on a B200: the kernels that replace an ordered f32 reduction by a parallel tree,
checked against the CPU oracle (which keeps the reference's order) with a tolerance.

What must stay exact in fast mode and is checked as such: int8 quantisation given the same
input, cache and state bytes written by unchanged kernels, the argmax rule.  What may move by
f32 rounding: rms_norm's rstd, a GEMV row's sum over blocks, the attention softmax sums.

Bars.  Per operator: a few f32 roundings (GEMV), one bf16 step on near-ties (norm, attention).
Whole model: greedy tokens identical wherever the oracle's top-1/top-2 margin exceeds twice the
observed logit difference.  Logits: max_abs 1e-2 is out of reach for any reordering on random-init
weights (at Qwen3.5-4B size by a factor of 40, on the eight-layer test model by a few): the forward re-quantises
activations to int8 some 230 times, so a last-bit difference that moves one bf16 rounding becomes
a whole quantisation step downstream and the difference settles at the quantisation-noise level.
The reference itself shows it: its two accumulate variants (fused multiply-add on the SDOT paths,
multiply-then-add in the portable fallback, Q8Scalar.cpp:192-199) differ by max_abs 0.3-0.4
(rms 0.07, logit std 1.0) on this model.  The full-size bar is therefore: the fast mode stays
within 1.5 x the spread between the reference's own two variants, measured on the same positions.
"""
import ctypes as C

import numpy as np
import pytest

import llmcp_b200 as L
import oracle

pytestmark = pytest.mark.gpu
f = oracle.bf16_to_f32


def bf16(a):
    return oracle.f32_to_bf16(np.asarray(a, dtype=np.float32))


@pytest.fixture
def fast_mode():
    L.set_mode("fast")
    yield
    L.set_mode("exact")


def bf16_ulps(got, want):
    """Distance in bf16 steps between two arrays of bf16 bit patterns (same sign assumed near zero)."""
    g = got.astype(np.int32)
    w = want.astype(np.int32)
    g = np.where(g & 0x8000, 0x8000 - g, g)
    w = np.where(w & 0x8000, 0x8000 - w, w)
    return np.abs(g - w)


@pytest.mark.parametrize("M,H", [(1, 2560), (3, 2560), (1, 64), (5, 4096), (2, 8192)])
def test_rms_norm_fast(fast_mode, M, H):
    rng = np.random.default_rng(H + M)
    x = bf16(rng.standard_normal((M, H)) * rng.choice([0.01, 1.0, 50.0], size=(M, 1)))
    w = bf16(rng.standard_normal(H) * 0.1)
    got = L.ops.rms_norm(x, w)
    want = oracle.rms_norm(x, w)
    ulps = bf16_ulps(got, want)
    # rstd may differ in its last f32 bit, which moves a bf16 rounding only on a near-tie
    assert ulps.max() <= 1 and (ulps != 0).mean() < 0.01, (ulps.max(), (ulps != 0).mean())


@pytest.mark.parametrize("N,K", [(9216, 2560), (2560, 9216), (2560, 4096), (12352 // 16 * 16, 2560), (1024, 2560), (248, 4096)])
def test_gemv_fast_reduction(N, K):
    """flags 16: tree-reduced row sums; against the oracle's ascending fma chain."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(N + K)
    w = (rng.standard_normal((N, K)) * 0.02).astype(np.float32)
    packed = oracle.pack_q8_0_p4(w)
    x = bf16(rng.standard_normal((1, K)))
    want = oracle.linear_q8(x, packed, N, y_bf16=False)[0]
    lib = L.lib()
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    ptr = lambda t: C.c_void_p(t.data_ptr())
    records = torch.from_numpy(packed).cuda()
    wq = torch.empty((N, K), dtype=torch.int8, device="cuda")
    wd = torch.empty((N, K // 32), dtype=torch.float16, device="cuda")
    assert lib.llmcp_dev_repack_q8(ptr(records), C.c_int64(N), C.c_int64(K), ptr(wq), ptr(wd), stream) == 0
    xd = torch.from_numpy(x.view(np.int16)).cuda()
    aq = torch.empty(K, dtype=torch.int8, device="cuda")
    scales = torch.empty(K // 32, dtype=torch.float32, device="cuda")
    assert lib.llmcp_dev_act_quant(ptr(xd), 1, C.c_int64(1), C.c_int64(K), ptr(aq), ptr(scales), stream) == 0
    bound = 4e-6 * float(np.abs(want).max()) + 1e-7  # a few f32 roundings of the largest term
    for flags in (16, 17, 19):
        y = torch.full((N,), float("nan"), dtype=torch.float32, device="cuda")
        rc = lib.llmcp_dev_gemv_q8(ptr(aq), ptr(scales), C.c_int64(K), ptr(wq), ptr(wd), C.c_int64(N), ptr(y), 0, 0, 0,
                                   flags, stream)
        assert rc == 0, L.last_error()
        torch.cuda.synchronize()
        got = y.cpu().numpy()
        assert np.isfinite(got).all()
        assert np.abs(got - want).max() <= bound, (flags, np.abs(got - want).max(), bound)


@pytest.mark.parametrize("nh,nkv,hd,position", [(16, 4, 256, 0), (16, 4, 256, 31), (16, 4, 256, 32), (16, 4, 256, 1030),
                                               (4, 2, 256, 77), (8, 4, 128, 200), (4, 4, 128, 65)])
def test_attention_decode_fast(fast_mode, nh, nkv, hd, position):
    rng = np.random.default_rng(position + nh)
    rot, cap = 64, position + 9
    qg = bf16(rng.standard_normal((1, nh * 2 * hd)))
    k = bf16(rng.standard_normal((1, nkv * hd)))
    v = bf16(rng.standard_normal((1, nkv * hd)))
    qn = bf16(rng.standard_normal(hd) * 0.1)
    kn = bf16(rng.standard_normal(hd) * 0.1)
    cos, sin = L.make_cos_sin(position, rot, 1e7)
    cache = bf16(rng.standard_normal((2, nkv, cap, hd)))
    got, got_cache = L.ops.attention(qg, k, v, qn, kn, cos[None], sin[None], cache, position, nh, nkv, hd, rot)
    want, want_cache = oracle.attention(qg, k, v, qn, kn, cos[None], sin[None], cache, position, nh, nkv, hd, rot)
    # cached rows other than the new one are untouched; the new key row may move by a bf16 step on
    # a near-tie (tree-summed norm), the new value row is a copy
    cache_ulps = bf16_ulps(got_cache, want_cache)
    assert cache_ulps.max() <= 1 and np.count_nonzero(cache_ulps) <= nkv * hd // 20
    assert np.array_equal(got_cache[1], want_cache[1])
    assert np.array_equal(np.delete(got_cache[0], position, axis=1), np.delete(want_cache[0], position, axis=1))
    ulps = bf16_ulps(got, want)
    assert np.isfinite(f(got)).all()
    assert ulps.max() <= 2 and (ulps != 0).mean() < 0.05, (ulps.max(), (ulps != 0).mean())


def test_attention_decode_fast_long_context(fast_mode):
    """8192 cached keys: several 32-key tiles per split."""
    rng = np.random.default_rng(8192)
    nh, nkv, hd, rot, position = 16, 4, 256, 64, 8192
    cap = position + 1
    qg = bf16(rng.standard_normal((1, nh * 2 * hd)))
    k = bf16(rng.standard_normal((1, nkv * hd)))
    v = bf16(rng.standard_normal((1, nkv * hd)))
    norm = np.zeros(hd, np.uint16)
    cos, sin = L.make_cos_sin(position, rot, 1e7)
    cache = bf16(rng.standard_normal((2, nkv, cap, hd)))
    got, _ = L.ops.attention(qg, k, v, norm, norm, cos[None], sin[None], cache, position, nh, nkv, hd, rot)
    want, _ = oracle.attention(qg, k, v, norm, norm, cos[None], sin[None], cache, position, nh, nkv, hd, rot)
    ulps = bf16_ulps(got, want)
    # 65 partial results per head are merged in another order than the key order: a bf16 step or two
    # where that moves a rounding; more steps only on outputs that cancel to nearly zero
    error, scale = np.abs(f(got) - f(want)), np.abs(f(want)).max()
    assert ((ulps <= 2) | (error <= scale * 2.0 ** -9)).all(), (ulps.max(), error.max(), scale)
    assert (ulps != 0).mean() < 0.05, (ulps != 0).mean()


@pytest.mark.parametrize("S,position", [(130, 0), (64, 0), (2, 0), (300, 0), (70, 64), (129, 7), (1024, 0)])
def test_attention_prefill_on_tensor_cores(fast_mode, S, position):
    """More than one query token in fast mode: Q K^T and P V on the tensor cores with the softmax
    weights rounded to bf16.  Against the oracle (f32 weights, key-ordered sums): every output within
    2^-7 of the largest one, nearly all within two bf16 steps; the cache as in the one-token test."""
    rng = np.random.default_rng(S * 31 + position)
    nh, nkv, hd, rot = 16, 4, 256, 64
    cap = position + S + 5
    qg = bf16(rng.standard_normal((S, nh * 2 * hd)))
    k = bf16(rng.standard_normal((S, nkv * hd)))
    v = bf16(rng.standard_normal((S, nkv * hd)))
    qn = bf16(rng.standard_normal(hd) * 0.1)
    kn = bf16(rng.standard_normal(hd) * 0.1)
    rows = [L.make_cos_sin(position + t, rot, 1e7) for t in range(S)]
    cos, sin = np.stack([r[0] for r in rows]), np.stack([r[1] for r in rows])
    cache = bf16(rng.standard_normal((2, nkv, cap, hd)))
    got, got_cache = L.ops.attention(qg, k, v, qn, kn, cos, sin, cache, position, nh, nkv, hd, rot)
    want, want_cache = oracle.attention(qg, k, v, qn, kn, cos, sin, cache, position, nh, nkv, hd, rot)
    cache_ulps = bf16_ulps(got_cache, want_cache)
    assert cache_ulps.max() <= 1 and np.count_nonzero(cache_ulps) <= S * nkv * hd // 20
    assert np.array_equal(got_cache[1], want_cache[1])
    assert np.isfinite(f(got)).all()
    error, scale = np.abs(f(got) - f(want)), np.abs(f(want)).max()
    ulps = bf16_ulps(got, want)
    assert error.max() <= scale * 2.0 ** -7, (error.max(), scale)
    assert ((ulps <= 2) | (error <= scale * 2.0 ** -9)).mean() > 0.999, ((ulps > 2).mean(), error.max(), scale)


@pytest.mark.parametrize("S,nk,nv", [(64, 16, 32), (1024, 16, 32), (33, 16, 16), (2, 2, 8)])
def test_gated_delta_net_prefill_fast(fast_mode, S, nk, nv):
    """Prefill recurrence with the state rows of two columns split over eight lanes and fused multiply-adds:
    against the oracle, outputs within a bf16 step or two, the final state to f32 rounding noise, and
    the golden vectors within the reference's own tolerance."""
    dk = dv = 128
    rng = np.random.default_rng(S + nv)
    channels = 2 * nk * dk + nv * dv
    conv, a = bf16(rng.standard_normal((S, channels))), bf16(rng.standard_normal((S, nv)))
    b = bf16(rng.standard_normal((S, nv)))
    a_log = (rng.standard_normal(nv) * 0.2).astype(np.float32)
    dt = bf16(rng.standard_normal(nv) * 0.2)
    state = (rng.standard_normal((nv, dk, dv)) * 0.1).astype(np.float32)
    got, got_state = L.ops.gated_delta_net(conv, a, b, a_log, dt, state, nk, nv, dk, dv)
    want, want_state = oracle.gated_delta_net(conv, a, b, a_log, dt, state, nk, nv, dk, dv)
    assert np.isfinite(f(got)).all() and np.isfinite(got_state).all()
    ulps = bf16_ulps(got, want)
    error, scale = np.abs(f(got) - f(want)), np.abs(f(want)).max()
    assert ((ulps <= 2) | (error <= scale * 2.0 ** -9)).all(), (ulps.max(), error.max(), scale)
    assert (ulps != 0).mean() < 0.05, (ulps != 0).mean()
    assert np.abs(got_state - want_state).max() <= 1e-4 * np.abs(want_state).max()


SMALL = dict(hidden=256, intermediate=512, vocab=2048, layers=8, full_interval=4, heads=4, kv_heads=2,
             head_dim=256, rotary=64, lin_k_heads=2, lin_v_heads=8, lin_k_dim=128, lin_v_dim=128, conv_kernel=4)


def oracle_dims(d):
    return dict(full_interval=d.full_interval, heads=d.heads, kv_heads=d.kv_heads, head_dim=d.head_dim,
                rotary=d.rotary, lin_k_heads=d.lin_k_heads, lin_v_heads=d.lin_v_heads, lin_k_dim=d.lin_k_dim,
                lin_v_dim=d.lin_v_dim, conv_kernel=d.conv_kernel)


def compare_fast_with_oracle(dims, seed, prompt, steps, capacity, spread=False):
    """Teacher-forced comparison: both sides are fed the oracle's greedy tokens, so one flipped
    token does not derail the rest; returns (max |dlogit|, min margin, tokens that differed) and,
    with spread, also (rms dlogit, max and rms of the oracle's muladd variant against its fma one)."""
    data = L.synthetic_container(dims, seed)
    arena = L.Arena().from_buffer(data)
    model = oracle.Model(data, arena.manifest, oracle_dims(dims))
    state = model.new_state(capacity)
    other = oracle.Model(data, arena.manifest, oracle_dims(dims), mode="muladd") if spread else None
    other_state = other.new_state(capacity) if spread else None
    sq, other_worst, other_sq, count = 0.0, 0.0, 0.0, 0
    engine = L.Engine(data, dims, capacity=capacity, mode="fast")
    exact = L.Engine(data, dims, capacity=capacity, mode="exact")
    tokens, pos = list(prompt), 0
    worst, margins, flips = 0.0, [], []
    for step in range(steps + 1):
        got, got_token = engine.forward(tokens, pos)
        ref, ref_token = exact.forward(tokens, pos)
        want = model.forward(state, tokens, pos)
        assert np.array_equal(ref.view(np.uint32), want.view(np.uint32)), "exact mode must still match bit for bit"
        assert np.isfinite(got).all()
        diff = float(np.abs(got - want).max())
        worst = max(worst, diff)
        if spread:
            alt = other.forward(other_state, tokens, pos)
            other_worst = max(other_worst, float(np.abs(alt - want).max()))
            sq += float(np.square(got - want, dtype=np.float64).sum())
            other_sq += float(np.square(alt - want, dtype=np.float64).sum())
            count += got.size
        margin = oracle.top2_margin(want)
        margins.append(margin)
        want_token = oracle.argmax(want)
        if got_token != want_token:
            flips.append((step, margin, diff))
            assert margin <= 2 * diff, f"token differs at step {step} although margin {margin} > 2 x {diff}"
        pos += len(tokens)
        tokens = [want_token]
    engine.close()
    exact.close()
    model.close()
    if spread:
        other.close()
        return worst, min(margins), flips, (sq / count) ** 0.5, other_worst, (other_sq / count) ** 0.5
    return worst, min(margins), flips


def test_fast_model_matches_oracle_within_tolerance():
    d = L.default_dims().copy(**SMALL)
    worst, margin, flips, rms, ref_worst, ref_rms = compare_fast_with_oracle(
        d, 20261125, [17, 5, 900, 2047, 0, 33, 33, 1200], steps=24, capacity=40, spread=True)
    print(f"fast vs oracle: max |dlogit| {worst:.3e} rms {rms:.3e}; reference muladd vs fma: max {ref_worst:.3e} "
          f"rms {ref_rms:.3e}; min top-2 margin {margin:.3e}, flips {flips}")
    # 1e-2 where the model is tame enough, else the spread of the reference's own two variants
    assert worst <= max(1e-2, 1.5 * ref_worst) and rms <= max(1e-3, 1.5 * ref_rms)


def test_fast_generate_is_deterministic_and_matches_forward():
    """The device-resident loop (CUDA graph) and the call-by-call path of a fast engine agree bit
    for bit with each other: the mode changes the order of additions, not their determinism."""
    d = L.default_dims().copy(**SMALL)
    data = L.synthetic_container(d, 3)
    a = L.Engine(data, d, capacity=40, mode="fast")
    b = L.Engine(data, d, capacity=40, mode="fast")
    prompt = [1, 2, 3, 4, 5]
    _, first = a.forward(prompt, 0)
    _, first_b = b.forward(prompt, 0)
    assert first == first_b
    generated, _ = a.generate(first, len(prompt), 12)
    tokens, pos, token = [], len(prompt), first
    for _ in range(12):
        _, token = b.forward([token], pos)
        tokens.append(token)
        pos += 1
    assert generated.tolist() == tokens
    a.close()
    b.close()


@pytest.mark.slow
def test_fast_full_size_model():
    """Qwen3.5-4B dimensions: 24-token prefill and 6 teacher-forced steps in fast mode, held to
    the spread between the reference's own two accumulate variants (see the module docstring)."""
    d = L.default_dims()
    worst, margin, flips, rms, ref_worst, ref_rms = compare_fast_with_oracle(d, 20261125, [9419] * 24, steps=6, capacity=40,
                                                                           spread=True)
    print(f"full size, fast vs oracle: max |dlogit| {worst:.3e} rms {rms:.3e}; the reference's muladd variant vs its "
          f"fma variant: max {ref_worst:.3e} rms {ref_rms:.3e}; min top-2 margin {margin:.3e}, flips {flips}")
    assert worst <= 1.5 * ref_worst and rms <= 1.5 * ref_rms
