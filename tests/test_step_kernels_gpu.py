"""Kernels chosen by size: each at the edges of its range against float64."""
import pytest
import torch

from rvllm_b200.errors import KernelError
from rvllm_b200.kernels import get_library

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def K():
    return get_library("cuda:0")


def rel_err(a, ref):
    return float((a.double().cpu() - ref).abs().max() / ref.abs().max().clamp(min=1e-30))


@pytest.mark.parametrize("N,Kd", [(17, 32), (130, 512), (300, 516), (64, 1028), (129, 2052), (40, 30), (5000, 96), (16, 4100),
                                  (64, 64), (250, 64), (16, 512)])
def test_gemm_f32_rows_do_not_depend_on_the_batch(K, N, Kd):
    """Few rows take the streaming kernel (in six sizes), more the tiles with K over 1, 2 or 4 CTAs: one order of summation, so
    the same bits; K with short last segments, fewer segments than 16, and rows that are not whole 16-byte words."""
    torch.manual_seed(N + Kd)
    x = torch.randn(300, Kd, device="cuda")
    w = torch.randn(N, Kd, device="cuda")
    b, r = torch.randn(N, device="cuda"), torch.randn(300, N, device="cuda")
    ref = x.double().cpu() @ w.double().cpu().t() + b.double().cpu() + r.double().cpu()
    whole = K.linear(x, w, b, r)
    # a segment is a chain of at most K / 16 + 32 roundings of 2^-24 each, on sums of about sqrt(K): far below 3e-6 of the largest value
    assert rel_err(whole, ref) < 3e-6
    for M in (1, 2, 3, 4, 5, 8, 9, 16, 17, 32, 33, 128, 129):
        assert torch.equal(K.linear(x[:M].contiguous(), w, b, r[:M].contiguous()), whole[:M]), M
    shifted = torch.empty(5 * Kd + 1, device="cuda")[1:].view(5, Kd).copy_(x[:5])        # not on a 16-byte boundary
    assert torch.equal(K.linear(shifted, w, b, r[:5].contiguous()), whole[:5])


@pytest.mark.parametrize("rows,cols,y_dtype", [(3, 4, torch.float32), (2, 1028, torch.bfloat16), (5, 4096, torch.float32), (2, 16384, torch.float32),
                                               (2, 16388, torch.bfloat16), (3, 130, torch.float32)])
def test_stream_norms_in_words_of_four(K, rows, cols, y_dtype):
    """Rows in registers (whole words of four, up to 16,384 columns) and rows read again: the same sums and norms."""
    torch.manual_seed(cols)
    y = torch.randn(rows, cols, device="cuda").to(y_dtype)
    x = torch.randn(rows, cols, device="cuda")
    g, g2 = torch.randn(cols, device="cuda"), torch.randn(cols, device="cuda").bfloat16()
    rms = lambda v, w, e: v / (v.square().mean(-1, keepdim=True) + e).sqrt() * w.double().cpu()      # noqa: E731
    new = x.double().cpu() + rms(y.double().cpu(), g, 1e-5)
    got, nxt = K.residual_rmsnorm(y, g, 1e-5, x.clone(), torch.float32, next_norm=(g2, 1e-6))
    # float sums of `cols` squares in a tree: a few 2^-24 times log2(cols)
    assert rel_err(got, new) < 2e-6 and rel_err(nxt, rms(new, g2, 1e-6)) < 4e-6
    got, same = K.residual_rmsnorm(y, g, 1e-5, None, torch.bfloat16)
    assert rel_err(got, rms(y.double().cpu(), g, 1e-5)) < 2e-6 and torch.equal(same, got.bfloat16())
    if y_dtype == torch.float32:
        got, nxt = K.stream_add_norm(x.clone(), y, (g, 1e-5), torch.float32)
        want = x.double().cpu() + y.double().cpu()
        assert rel_err(got, want) < 2e-7 and rel_err(nxt, rms(want, g, 1e-5)) < 4e-6


@pytest.mark.parametrize("T,E,top,ff,width,gated,identity", [(1, 8, 2, 32, 64, True, False), (7, 5, 3, 96, 160, False, True), (33, 40, 4, 160, 96, True, False),
                                                             (100, 3, 2, 64, 96, True, False), (9, 70, 4, 1408, 2048, False, False),
                                                             (100, 12, 8, 64, 96, True, True), (127, 9, 16, 32, 64, False, False)])
def test_moe_of_few_tokens_on_the_tensor_cores(K, T, E, top, ff, width, gated, identity):
    """Every expert's pairs as the columns of one product: lists of one to many pairs (several passes), numbers that name
    nobody (-1) or the token itself, rows of 16 that end inside the matrix, sums of more pairs than shared memory holds at a
    time (from about 620 on); and a token's bits do not depend on the others."""
    torch.manual_seed(T * E)
    gu = (torch.randn(E, (2 if gated else 1) * ff, width, device="cuda") * 0.1).bfloat16()
    dn = (torch.randn(E, width, ff, device="cuda") * 0.1).bfloat16()
    x = torch.randn(T, width, device="cuda").bfloat16()
    ch = torch.randint(-1, E + (2 if identity else 0), (T, top), device="cuda", dtype=torch.int32)
    w, add, scale = torch.rand(T, top, device="cuda"), torch.randn(T, width, device="cuda"), torch.rand(T, device="cuda")
    run = lambda n: K.moe_experts(x[:n].contiguous(), ch[:n].contiguous(), gu, dn, 0.5, add=add[:n].contiguous(), out_dtype=torch.float32,      # noqa: E731
                                  weights=w[:n].contiguous(), activation="silu" if gated else "relu2", add_scale=scale[:n].contiguous(), identity=identity)
    out, ref = run(T), (scale[:, None] * add).double().cpu()
    for t in range(T):
        for k in range(top):
            e = int(ch[t, k])
            if e >= E:
                ref[t] += 0.5 * float(w[t, k]) * x[t].double().cpu()
            if not 0 <= e < E:
                continue
            h = gu[e].double().cpu() @ x[t].double().cpu()
            a = torch.nn.functional.silu(h[:ff]) * h[ff:] if gated else torch.relu(h) ** 2
            ref[t] += 0.5 * float(w[t, k]) * (dn[e].double().cpu() @ a)
    assert rel_err(out, ref) < 4e-3                          # the activations are rounded to bfloat16 (2^-9) before the second product
    assert torch.equal(run(1), out[:1])


@pytest.mark.parametrize("T,E,top,ff,width", [(8, 8, 2, 4096, 1024), (33, 16, 4, 1408, 2048), (20, 16, 4, 256, 1024)])
def test_moe_sums_of_whole_activations(K, T, E, top, ff, width):
    """Activations that are whole numbers of at most 256 (squares of sums of few ones and twos) are the same in bfloat16, so
    what is left is the error of the float sums over ff and the slots."""
    torch.manual_seed(T)
    gu = (torch.randint(-2, 3, (E, ff, width), device="cuda") * (torch.rand(E, ff, width, device="cuda") < 4.0 / width)).bfloat16()
    x, dn = torch.randint(0, 2, (T, width), device="cuda").bfloat16(), (torch.randn(E, width, ff, device="cuda") * 0.02).bfloat16()
    ch = torch.stack([torch.randperm(E, device="cuda")[:top] for _ in range(T)]).to(torch.int32)
    w = torch.rand(T, top, device="cuda")
    out = K.moe_experts(x, ch, gu, dn, 1.0, out_dtype=torch.float32, weights=w, activation="relu2")
    ref = torch.zeros(T, width, dtype=torch.float64, device="cuda")
    for e in range(E):
        h = torch.relu(x.double() @ gu[e].double().t()) ** 2
        assert h.max() <= 256
        ref += (h @ dn[e].double().t()) * (w.double() * (ch == e)).sum(1, keepdim=True)
    # 2-norms: a float's own rounding is up to 2^-24 / sqrt(3) = 3.4e-8; the sums of 128 k add less than that again
    # (float chains, one pair at a time: 4.2e-8 to 5.8e-8; one accumulator of the tensor cores through all of k: up to 7.5e-8)
    assert float((out.double() - ref).norm() / ref.norm()) < 5e-8


@pytest.mark.parametrize("M,N,Kd", [(130, 264, 72), (300, 96, 128), (512, 512, 4096), (5, 200, 136), (64, 1024, 264), (200, 130, 72), (5, 1024, 4096)])
@pytest.mark.parametrize("bias_dtype", [torch.float32, torch.bfloat16])
def test_bias_and_clamped_gate_in_the_products_epilogues(K, M, N, Kd, bias_dtype):
    """Plain, residual and clamp-gated products with a bias: both GEMMs, one CTA, pairs, K split over a cluster and (few gated rows of
    a long K) over CTAs that meet in scratch memory."""
    assert (M, Kd) != (5, 4096) or K.gemm_splits((N // 2 + 63) // 64, Kd) > 1
    torch.manual_seed(M + N)
    x, w = torch.randn(M, Kd, device="cuda").bfloat16(), (torch.randn(N, Kd, device="cuda") * 0.1).bfloat16()
    b, r = torch.randn(N, device="cuda").to(bias_dtype), torch.randn(M, N, device="cuda").bfloat16()
    ref = x.double().cpu() @ w.double().cpu().t() + b.double().cpu()
    assert rel_err(K.linear(x, w, b, None, torch.float32), ref) < 2e-5      # float sums of exact products
    if N % 8 == 0:
        assert rel_err(K.linear(x, w, b, r), ref + r.double().cpu()) < 5e-3      # one rounding to bfloat16
    half = N // 2
    gate, up = ref[:, :half].clamp(max=2.0), ref[:, half:].clamp(-2.0, 2.0)
    want = gate * torch.sigmoid(1.7 * gate) * (up + 1)
    assert rel_err(K.gate_up_clamp(x, w, b, 2.0, 1.7), want) < 5e-3


@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("form", ["float64", "strided", "one value", "strided residual", "one residual row", "odd address", "odd residual", "no multiple of 8"])
def test_biases_and_residuals_that_no_epilogue_takes(K, form, out_dtype):
    """Types, strides, addresses and shapes that broadcast: what the library's product takes beside a bias, and a clamped gate too."""
    torch.manual_seed(4)
    M, N, Kd = 300, 130 if form == "no multiple of 8" else 96, 128
    x, w = torch.randn(M, Kd, device="cuda").bfloat16(), (torch.randn(N, Kd, device="cuda") * 0.1).bfloat16()
    b, r = torch.randn(N, device="cuda"), torch.randn(M, N, device="cuda").bfloat16()
    if form == "float64":
        b = b.double()
    elif form == "strided":
        b = torch.randn(2 * N, device="cuda")[::2]
    elif form == "one value":
        b = b[:1]
    elif form == "strided residual":
        r = torch.randn(M, 2 * N, device="cuda").bfloat16()[:, ::2]
    elif form == "one residual row":
        r = r[:1]
    elif form == "odd address":
        x = torch.randn(M * Kd + 1, device="cuda").bfloat16()[1:].view(M, Kd)
    elif form == "odd residual":
        r = torch.randn(M * N + 1, device="cuda").bfloat16()[1:].view(M, N)
    ref = x.double().cpu() @ w.double().cpu().t() + b.double().cpu()
    tol = 2e-5 if out_dtype == torch.float32 else 1e-2      # float sums; two roundings to bfloat16 where the bias is one
    assert rel_err(K.linear(x, w, b, None, out_dtype), ref) < tol
    if out_dtype == torch.bfloat16:
        assert rel_err(K.linear(x, w, b, r, out_dtype), ref + r.double().cpu()) < tol
    gate, up = ref[:, :N // 2].clamp(max=2.0), ref[:, N // 2:].clamp(-2.0, 2.0)
    assert rel_err(K.gate_up_clamp(x, w, b, 2.0, 1.7), gate * torch.sigmoid(1.7 * gate) * (up + 1)) < 5e-3
    for m in (4, M):                                        # a weight of fewer columns is refused, whatever the path
        with pytest.raises(KernelError):
            K.gate_up_clamp(x[:m].clone(), w[:, :64].contiguous(), torch.randn(N, device="cuda"), 2.0, 1.7)


@pytest.mark.parametrize("heads,P,N,groups,lens", [(4, 64, 128, 2, (33, 1, 64, 65)), (6, 48, 64, 3, (130, 2)), (2, 80, 128, 1, (40,)), (2, 16, 64, 1, (200,))])
def test_ssm_scan_in_chunks(K, heads, P, N, groups, lens, monkeypatch):
    """The chunked form against the recurrence in float64: portions that end inside a chunk, single tokens, a padding row, column
    blocks that are not full, a state to continue from, decays from weak to total."""
    torch.manual_seed(P)
    T, C = sum(lens), heads * P + 2 * groups * N
    xbc = torch.randn(T, C, device="cuda").bfloat16()
    proj = torch.randn(T, heads + 3, device="cuda") * 2
    bias, a_log, D = torch.randn(heads, device="cuda") - 2, torch.linspace(-2, 3, heads, device="cuda"), torch.randn(heads, device="cuda")
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    slots = list(range(len(lens)))
    if len(lens) > 2:
        slots[1] = -1
    state = torch.randn(len(lens), heads * N * P + 8, device="cuda")
    S = state[:, :heads * N * P].double().cpu().view(-1, heads, N, P).clone()
    xd = xbc.double().cpu()
    x, B, Cm = xd[:, :heads * P].view(T, heads, P), xd[:, heads * P:heads * P + groups * N].view(T, groups, N), xd[:, heads * P + groups * N:].view(T, groups, N)
    dt = torch.nn.functional.softplus((proj[:, 3:] + bias).double().cpu())
    a = torch.exp(-torch.exp(a_log.double().cpu()) * dt)
    want, rep = torch.zeros(T, heads, P, dtype=torch.float64), heads // groups
    for s, slot in enumerate(slots):
        for t in range(cu[s], cu[s + 1]):
            if slot >= 0:
                S[s] = a[t][:, None, None] * S[s] + (dt[t][:, None] * B[t].repeat_interleave(rep, 0))[:, :, None] * x[t][:, None, :]
                want[t] = torch.einsum("hn,hnp->hp", Cm[t].repeat_interleave(rep, 0), S[s]) + D.double().cpu()[:, None] * x[t]
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")      # noqa: E731
    walked = state.clone()
    run = lambda st, chunked: K.ssm_scan(xbc, proj, 3, bias, a_log, D, i32(cu), i32(slots), st, heads, P, N, groups, max_q_len=max(lens), chunked=chunked)      # noqa: E731
    used, load = [], K._lib
    monkeypatch.setattr(K, "_lib", lambda source, *a: used.append(source) or load(source, *a))
    got, walk = run(state, True), run(walked, False)
    assert used == ["ssm_chunk.cu", "ssm.cu"]
    # three bfloat16 terms hold a float: the error is that of float sums over N and 64 products
    assert rel_err(got, want.view(T, -1)) < 2e-6
    assert rel_err(state[:, :heads * N * P], S.view(len(lens), -1)) < 2e-6
    # ... and no larger than that of the sums token by token, but for the last rounding of a float (2^-24 over sqrt(3) in 2-norms)
    norm = lambda a, ref: float((a.double().cpu() - ref).norm() / ref.norm())      # noqa: E731
    assert norm(got, want.view(T, -1)) <= norm(walk, want.view(T, -1)) + 3.5e-8
    assert norm(state[:, :heads * N * P], S.view(len(lens), -1)) <= norm(walked[:, :heads * N * P], S.view(len(lens), -1)) + 3.5e-8


@pytest.mark.parametrize("N,lens", [(128, (1, 40, 5, 64, 31)), (64, (32, 1, 1)), (128, (33, 33))])
def test_ssm_scan_bits_depend_on_the_request_alone(K, N, lens, monkeypatch):
    """Long portions of a step go chunk by chunk and short ones beside them token by token, each with the bits that it has alone;
    a padding row (slot -1) leaves no state and reads as zero."""
    torch.manual_seed(N + len(lens))
    heads, P, T = 4, 48, sum(lens)
    xbc = torch.randn(T, heads * P + 2 * N, device="cuda").bfloat16()
    proj, bias = torch.randn(T, heads, device="cuda"), torch.randn(heads, device="cuda") - 2
    a_log, D = torch.linspace(-1, 2, heads, device="cuda"), torch.randn(heads, device="cuda")
    before = torch.randn(len(lens), heads * N * P, device="cuda")
    cu = torch.tensor((0,) + lens).cumsum(0).tolist()
    slots = list(range(len(lens)))
    if len(lens) > 2:
        slots[2] = -1
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")      # noqa: E731

    def run(a, b, cu, slots):
        state = before.clone()
        return K.ssm_scan(xbc[a:b].contiguous(), proj[a:b].contiguous(), 0, bias, a_log, D, i32(cu), i32(slots), state, heads, P, N, 1,
                          max_q_len=max(v - u for u, v in zip(cu, cu[1:]))), state
    used, load = [], K._lib
    monkeypatch.setattr(K, "_lib", lambda source, *a: used.append(source) or load(source, *a))
    whole, state = run(0, T, cu, slots)
    assert used == (["ssm_chunk.cu"] if len(set(lens)) == 1 else ["ssm.cu", "ssm_chunk.cu"])
    for i, n in enumerate(lens):
        y, s = run(cu[i], cu[i + 1], [0, n], [slots[i]])
        assert used[-1] == ("ssm_chunk.cu" if n >= 32 else "ssm.cu")
        assert torch.equal(y, whole[cu[i]:cu[i + 1]]) and torch.equal(s[i], state[i])
        assert slots[i] >= 0 or (torch.equal(state[i], before[i]) and not y.any())


@pytest.mark.parametrize("heads,T,segments", [(2, 2816, False), (2, 2817, True), (8, 5000, True), (64, 5000, False), (300, 3000, False)])
def test_ssm_scan_of_few_heads_takes_segments(K, heads, T, segments, monkeypatch):
    """Long portions on few CTAs go in segments side by side where the chunks' walk is longer: the same values."""
    torch.manual_seed(heads)
    P, N = 16, 64
    xbc = torch.randn(T, heads * P + 2 * N, device="cuda").bfloat16()
    proj, bias = torch.randn(T, heads, device="cuda"), torch.randn(heads, device="cuda") - 4
    a_log, D = torch.rand(heads, device="cuda"), torch.randn(heads, device="cuda")
    before = torch.randn(1, heads * N * P, device="cuda")
    cu, slots = torch.tensor([0, T], dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    used, load = [], K._lib
    monkeypatch.setattr(K, "_lib", lambda source, *a: used.append(source) or load(source, *a))
    runs = []
    for chunked in (None, segments):
        state = before.clone()
        runs.append((K.ssm_scan(xbc, proj, 0, bias, a_log, D, cu, slots, state, heads, P, N, 1, max_q_len=T, chunked=chunked), state))
    assert used == ["ssm.cu" if segments else "ssm_chunk.cu", "ssm_chunk.cu" if segments else "ssm.cu"]
    # two orders of float sums along up to 5,000 tokens with decays near 1
    assert all(rel_err(a, b.double().cpu()) < 2e-5 for a, b in zip(*runs))


@pytest.mark.parametrize("N,value,where", [(128, float("inf"), 5), (64, float("nan"), 77), (128, float("-inf"), 64), (64, float("inf"), 129)])
@pytest.mark.parametrize("place", ["x", "B", "C", "dt"])
def test_ssm_scan_in_chunks_is_causal(K, N, value, where, place):
    """A number that is not finite reaches its own token and those after it, an x or a state its own column alone, as in the
    walk; the tokens before it, in its block of 16 and its chunk, and the other columns are what they are without it."""
    torch.manual_seed(N + where)
    heads, P, T = 2, 64, 130
    xbc = torch.randn(T, heads * P + 2 * N, device="cuda").bfloat16()
    proj, bias = torch.randn(T, heads, device="cuda"), torch.randn(heads, device="cuda") - 2
    a_log, D = torch.linspace(-1, 2, heads, device="cuda"), torch.randn(heads, device="cuda")
    state = torch.randn(1, heads * N * P, device="cuda")
    cu, slots = torch.tensor([0, T], dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    runs = []
    for odd in (True, False):
        target, column = (proj, 0) if place == "dt" else (xbc, {"x": 3, "B": heads * P + 9, "C": heads * P + N + 9}[place])
        target[where, column] = value if odd else 0.5
        state.view(heads, N, P)[1, 7, 40] = value if odd and place == "x" else 0.5
        for chunked in (True, False):
            s = state.clone()
            y = K.ssm_scan(xbc, proj, 0, bias, a_log, D, cu, slots, s, heads, P, N, 1, max_q_len=T, chunked=chunked)
            runs.append((y.view(T, heads, P), s.view(heads, N, P)))
    for got, walk in zip(runs[0], runs[1]):
        assert all(torch.equal(kind(got), kind(walk)) for kind in (torch.isnan, torch.isposinf, torch.isneginf))
    (y, s), _, (plain_y, plain_s), _ = runs
    assert rel_err(y[:where, 0], plain_y[:where, 0].double().cpu()) < 2e-6
    if place == "x":
        assert not y[where, 0, 3].isfinite()
        other = [p for p in range(P) if p != 3]
        assert rel_err(y[:, 0][:, other], plain_y[:, 0][:, other].double().cpu()) < 2e-6
        assert rel_err(s[0][:, other], plain_s[0][:, other].double().cpu()) < 2e-6


def test_ssm_scan_in_chunks_beside_a_step_size_that_dwarfs_the_others(K):
    """A sum of decays that one step of 10^17 dominates still tells the decays of the tokens after it."""
    torch.manual_seed(1)
    heads, P, N, T = 1, 16, 64, 64
    xbc, proj = torch.randn(T, heads * P + 2 * N, device="cuda").bfloat16(), torch.randn(T, heads, device="cuda")
    proj[20] = 1e17
    xbc[20, :P] = 0                                          # (what it brings is then nothing)
    zero, cu, slots = torch.zeros(heads, device="cuda"), torch.tensor([0, T], dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    runs = []
    for chunked in (True, False):
        state = torch.ones(1, heads * N * P, device="cuda")
        runs.append((K.ssm_scan(xbc, proj, 0, zero, zero, zero, cu, slots, state, heads, P, N, 1, max_q_len=T, chunked=chunked), state))
    for got, walk in zip(*runs):
        assert rel_err(got, walk.double().cpu()) < 2e-6


@pytest.mark.parametrize("inner,N,lens", [(70, 16, (1, 5, 16, 17, 35)), (33, 32, (18, 2)), (32, 16, (64,))])
def test_selective_scan_in_two_roles(K, inner, N, lens):
    torch.manual_seed(inner)
    T = sum(lens)
    u, z = torch.randn(T, inner, device="cuda"), torch.randn(T, inner + 4, device="cuda")
    raw, bias, A = torch.randn(T, inner, device="cuda"), torch.randn(inner, device="cuda"), -torch.rand(inner, N, device="cuda") * 4
    bc, D = torch.randn(T, 2 * N + 3, device="cuda"), torch.randn(inner, device="cuda")
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    state = torch.randn(len(lens), inner * N + 4, device="cuda")
    S = state[:, :inner * N].double().cpu().view(-1, inner, N).clone()
    dt, b64, u64 = torch.nn.functional.softplus((raw + bias).double().cpu()), bc.double().cpu(), u.double().cpu()
    want = torch.empty(T, inner, dtype=torch.float64)
    for s in range(len(lens)):
        for t in range(cu[s], cu[s + 1]):
            S[s] = torch.exp(dt[t][:, None] * A.double().cpu()) * S[s] + (dt[t] * u64[t])[:, None] * b64[t, 3:3 + N]
            want[t] = (S[s] * b64[t, 3 + N:]).sum(1) + D.double().cpu() * u64[t]
    want *= torch.nn.functional.silu(z[:, 4:].double().cpu())
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")      # noqa: E731
    got = K.selective_scan(u, raw, bias, A.contiguous(), bc, 3, 3 + N, D, z, 4, i32(cu), i32(list(range(len(lens)))), state, torch.float32, max_q_len=max(lens))
    assert rel_err(got, want) < 2e-6 and rel_err(state[:, :inner * N], S.view(len(lens), -1)) < 2e-6


@pytest.mark.parametrize("inner,N,lens", [(70, 16, (1, 5, 16, 17, 35)), (33, 32, (18, 2, 1, 1, 1, 1)), (40, 8, (1, 9)), (32, 16, (1,) * 26 + (40,))])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_selective_scan_bits_do_not_depend_on_the_step(K, inner, N, lens, dtype):
    """A request's outputs and state are the same bits alone, beside others and with its portion cut in two, whichever kernels the
    steps take; a padding row (slot -1) leaves no state."""
    torch.manual_seed(inner + N)
    T = sum(lens)
    u, z = torch.randn(T, inner, device="cuda").to(dtype), torch.randn(T, inner, device="cuda").to(dtype)
    raw, bias, A = torch.randn(T, inner, device="cuda"), torch.randn(inner, device="cuda"), (-torch.rand(inner, N, device="cuda") * 4).contiguous()
    bc, D = torch.randn(T, 2 * N, device="cuda"), torch.randn(inner, device="cuda")
    before = torch.randn(len(lens), inner * N, device="cuda")
    cu = torch.tensor((0,) + lens).cumsum(0).tolist()
    slots = list(range(len(lens)))
    slots[1] = -1
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")      # noqa: E731

    def run(a, b, cu, slots, state, longest):
        y = K.selective_scan(u[a:b].contiguous(), raw[a:b].contiguous(), bias, A, bc[a:b].contiguous(), 0, N, D, z[a:b].contiguous(), 0, i32(cu), i32(slots),
                             state, torch.float32, max_q_len=longest)
        return [y[cu[i]:cu[i + 1]] for i in range(len(slots)) if slots[i] >= 0], state
    whole, state = run(0, T, cu, slots, before.clone(), max(lens))
    for longest in (1, T, None):
        y, s = run(0, T, cu, slots, before.clone(), longest)
        assert all(map(torch.equal, y, whole)) and torch.equal(s, state)
    assert torch.equal(state[1], before[1])
    for i, y in zip([i for i in range(len(lens)) if slots[i] >= 0], whole):
        s = before.clone()
        for a, b in ((cu[i], cu[i] + 1), (cu[i] + 1, cu[i + 1])):
            if b > a:
                assert torch.equal(run(a, b, [0, b - a], [i], s, b - a)[0][0], y[a - cu[i]:b - cu[i]])
        assert torch.equal(s[i], state[i])


@pytest.mark.parametrize("taps,lens", [(4, (1, 1, 1)), (3, (2, 1)), (1, (1,)), (2, (1, 1)), (4, (2,))])
def test_convolution_of_single_tokens_in_one_launch(K, taps, lens):
    """One launch for the outputs and the state: the same as a long portion cut into these steps."""
    torch.manual_seed(taps)
    T, C = sum(lens), 131
    proj, w, b = torch.randn(T, C + 5, device="cuda"), torch.randn(C, taps, device="cuda"), torch.randn(C, device="cuda")
    state = torch.randn(len(lens) + 1, (taps - 1) * C + 7, device="cuda")
    hist = state[:, 7:].double().cpu().view(len(lens) + 1, taps - 1, C).clone()
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")      # noqa: E731
    seq = [s for s, n in enumerate(lens) for _ in range(n)]
    got = K.causal_conv_silu(proj, 5, C, w, b, i32(seq), i32(cu), i32(list(range(1, len(lens) + 1))), state, 7, torch.float32,
                             max_q_len=max(lens))
    for s, n in enumerate(lens):
        row = torch.cat([hist[s + 1], proj[cu[s]:cu[s + 1], 5:].double().cpu()])
        for t in range(n):
            v = b.double().cpu() + (row[t:t + taps] * w.double().cpu().t()).sum(0)
            assert rel_err(got[cu[s] + t], torch.nn.functional.silu(v)) < 2e-6
        assert taps == 1 or rel_err(state[s + 1, 7:], row[n:].reshape(-1)) < 1e-7


@pytest.mark.parametrize("taps,lens,in_dtype", [(4, (1, 2, 1, 2), torch.float32), (3, (2, 1), torch.bfloat16), (4, (1,) * 9 + (21,), torch.float32), (2, (2,), torch.bfloat16)])
def test_convolution_bits_do_not_depend_on_the_step(K, taps, lens, in_dtype):
    """A request's outputs and state are the same bits whatever runs beside it, and whichever of the two forms a step takes; a
    padding row (slot -1) starts from zeros and leaves no state."""
    torch.manual_seed(taps + len(lens))
    T, C = sum(lens), 131
    proj, w, b = torch.randn(T, C + 5, device="cuda").to(in_dtype), torch.randn(C, taps, device="cuda"), torch.randn(C, device="cuda")
    before = torch.randn(len(lens), (taps - 1) * C, device="cuda")
    cu = torch.tensor((0,) + lens).cumsum(0).tolist()
    slots = list(range(len(lens)))
    if len(lens) > 2:
        slots[1] = -1
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")      # noqa: E731

    def run(rows, which, longest):
        state = before.clone()
        n = [lens[s] for s in which]
        out = K.causal_conv_silu(proj[rows].contiguous(), 5, C, w, b, i32([i for i, k in enumerate(n) for _ in range(k)]),
                                 i32([0] + torch.tensor(n).cumsum(0).tolist()), i32([slots[s] for s in which]), state, 0, torch.float32, max_q_len=longest)
        return out, state
    whole, state = run(slice(0, T), range(len(lens)), max(lens))
    forms = [run(slice(0, T), range(len(lens)), longest) for longest in (2, 3, None)]
    assert all(torch.equal(whole, o) and torch.equal(state, s) for o, s in forms)
    for s in range(len(lens)):
        alone, own = run(slice(cu[s], cu[s + 1]), [s], lens[s])
        assert torch.equal(alone, whole[cu[s]:cu[s + 1]])
        assert torch.equal(own[s], state[s]) and (slots[s] >= 0 or torch.equal(state[s], before[s]))


@pytest.mark.parametrize("d,vd,heads,qk,lens", [(128, 128, 4, 2, (1, 15, 16, 17, 70)), (100, 36, 2, 1, (33,)), (64, 68, 2, 2, (20, 1)), (40, 4, 2, 1, (18,)),
                                                (128, 128, 4, 2, (1, 1, 1)), (100, 132, 2, 1, (2,)), (24, 8, 2, 2, (1, 2, 1))])
def test_delta_rule_of_portions_and_of_single_tokens(K, d, vd, heads, qk, lens):
    torch.manual_seed(d + vd)
    T = sum(lens)
    qkv, proj = torch.randn(T, 2 * qk * d + heads * vd, device="cuda"), torch.randn(T, 2 * heads + 1, device="cuda")
    a_log, bias = torch.randn(heads, device="cuda"), torch.randn(heads, device="cuda")
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    state = torch.randn(len(lens), heads * d * vd + 4, device="cuda")
    S = state[:, :heads * d * vd].double().cpu().view(-1, heads, d, vd).clone()
    f = qkv.double().cpu()
    rep = heads // qk
    q, k = (f[:, i * qk * d:(i + 1) * qk * d].view(T, qk, d).repeat_interleave(rep, 1) for i in (0, 1))
    v = f[:, 2 * qk * d:].view(T, heads, vd)
    q, k = q / (q.square().sum(-1, keepdim=True) + 1e-6).sqrt() * d ** -0.5, k / (k.square().sum(-1, keepdim=True) + 1e-6).sqrt()
    beta = torch.sigmoid(proj[:, 1:1 + heads].double().cpu())
    g = torch.exp(-torch.exp(a_log.double().cpu()) * torch.nn.functional.softplus((proj[:, 1 + heads:] + bias).double().cpu()))
    want = torch.empty(T, heads, vd, dtype=torch.float64)
    for s in range(len(lens)):
        for t in range(cu[s], cu[s + 1]):
            S[s] = g[t][:, None, None] * S[s]
            un = beta[t][:, None] * (v[t] - torch.einsum("hdv,hd->hv", S[s], k[t]))
            S[s] = S[s] + k[t][:, :, None] * un[:, None, :]
            want[t] = torch.einsum("hdv,hd->hv", S[s], q[t])
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")      # noqa: E731
    got = K.delta_rule(qkv, proj, 1, 1 + heads, a_log, bias, i32(cu), i32(list(range(len(lens)))), state, heads, qk, d, vd, 1e-6, max_q_len=max(lens))
    # float sums of d products along a chain of at most 70 tokens
    assert rel_err(got, want.view(T, -1)) < 3e-6 and rel_err(state[:, :heads * d * vd], S.view(len(lens), -1)) < 3e-6


@pytest.mark.parametrize("d,vd,heads,qk,lens", [(128, 128, 4, 2, (1, 40, 1, 2)), (100, 36, 2, 1, (2, 1, 3)), (64, 68, 2, 2, (1,) * 20 + (17,)), (40, 4, 2, 1, (19, 2)),
                                                (24, 8, 2, 2, (1, 5, 2)), (160, 8, 2, 1, (1, 9))])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_delta_rule_bits_do_not_depend_on_the_step(K, d, vd, heads, qk, lens, dtype):
    """A request's outputs and state are the same bits alone, beside others and with its portion cut in two, whichever kernels the
    steps take; a padding row (slot -1) leaves no state."""
    torch.manual_seed(d + vd)
    T = sum(lens)
    qkv, proj = torch.randn(T, 2 * qk * d + heads * vd, device="cuda").to(dtype), torch.randn(T, 2 * heads, device="cuda")
    a_log, bias = torch.randn(heads, device="cuda"), torch.randn(heads, device="cuda")
    before = torch.randn(len(lens), heads * d * vd, device="cuda")
    cu = torch.tensor((0,) + lens).cumsum(0).tolist()
    slots = list(range(len(lens)))
    slots[len(lens) // 2] = -1
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")      # noqa: E731

    def run(a, b, cu, slots, state, longest):
        o = K.delta_rule(qkv[a:b].contiguous(), proj[a:b].contiguous(), 0, heads, a_log, bias, i32(cu), i32(slots), state, heads, qk, d, vd, 1e-6, max_q_len=longest)
        return [o[cu[i]:cu[i + 1]] for i in range(len(slots)) if slots[i] >= 0], state
    whole, state = run(0, T, cu, slots, before.clone(), max(lens))
    for longest in (2, T, None):                            # the kernel of single tokens for all, the walk for all or beside it
        o, s = run(0, T, cu, slots, before.clone(), longest)
        assert all(map(torch.equal, o, whole)) and torch.equal(s, state)
    assert torch.equal(state[len(lens) // 2], before[len(lens) // 2])
    for i, o in zip([i for i in range(len(lens)) if slots[i] >= 0], whole):
        s = before.clone()
        for a, b in ((cu[i], cu[i] + 1), (cu[i] + 1, cu[i + 1])):
            if b > a:
                assert torch.equal(run(a, b, [0, b - a], [i], s, b - a)[0][0], o[a - cu[i]:b - cu[i]])
        assert torch.equal(s[i], state[i])

@pytest.mark.parametrize("d,vd,lens", [(128, 128, (33, 16, 20)), (64, 132, (17, 40, 8, 9)), (100, 36, (47,) * 12)])
def test_walks_of_two_and_of_four_columns_a_lane(K, d, vd, lens):
    """Steps whose blocks of two columns a lane are more than the SMs take four: the bits of each request alone, which takes two."""
    heads = 16
    torch.manual_seed(d + vd)
    T, N, W = sum(lens), len(lens), vd + 1
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert -(-vd // (16 if d > 64 else 32)) * heads * N > sms >= -(-W // (16 if d > 64 else 32)) * heads
    cu = torch.tensor((0,) + lens).cumsum(0).tolist()
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")      # noqa: E731
    qkv, gates = torch.randn(T, (2 * d + vd) * heads, device="cuda").bfloat16(), torch.randn(T, 2 * heads, device="cuda")
    proj = torch.cat([qkv.float(), gates], dim=1)
    a, b = torch.randn(heads, device="cuda"), torch.randn(heads, device="cuda")
    first = torch.randn(N, heads * d * vd, device="cuda")
    memory = torch.randn(N, heads * d * W + heads, device="cuda")

    def delta(i, j, cu, slots, s):
        return K.delta_rule(qkv[i:j].contiguous(), gates[i:j].contiguous(), 0, heads, a, b, i32(cu), i32(slots), s, heads, heads, d, vd, 1e-6, max_q_len=max(lens))

    def matrix(i, j, cu, slots, s):
        g0 = (2 * d + vd) * heads
        return torch.cat(K.mlstm_scan(proj[i:j].contiguous(), g0, g0 + heads, a, b + 2, i32(cu), i32(slots), s, heads, d, vd, 15.0, max_q_len=max(lens)), dim=1)
    for run, start in ((delta, first), (matrix, memory)):
        state = start.clone()
        whole = run(0, T, cu, list(range(N)), state)
        for n, (i, j) in enumerate(zip(cu, cu[1:])):
            own = start.clone()
            assert torch.equal(run(i, j, [0, j - i], [n], own), whole[i:j]) and torch.equal(own[n], state[n])


def test_talking_attention_on_eight_and_sixteen_warps(K):
    """The same tiles for twice the tokens a CTA: the same bits, and those of the attention's formula in float64."""
    import plain_tibepel as P
    from rvllm_b200.kernels.library import AttentionMeta
    torch.manual_seed(3)
    nh, nkv, hd, ps, T = 8, 4, 64, 16, 75
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")      # noqa: E731
    cache = torch.randn(5, nkv * ps * 2 * hd, device="cuda").bfloat16()
    meta = AttentionMeta(block_tables=i32([[3, 1, 0, 4, 2]]), cu_seqlens=i32([0, T]), ctx_lens=i32([T]), token_seq=i32([0] * T), slot_mapping=i32([0] * T),
                         num_seqs=1, max_q_len=T, max_ctx_len=T, page_size=ps)
    q = torch.randn(T, nh * hd, device="cuda").bfloat16()
    r, talk = torch.rand(nh, device="cuda"), torch.randn(nh, nh, device="cuda")
    out = []
    try:
        for K.TALKING_WARPS in (8, 16):
            out.append(K.talking_attention(q, cache, meta, None, nh, nkv, hd, hd, hd ** -0.5, r, r, talk, None))
    finally:
        del K.TALKING_WARPS
    assert torch.equal(*out)
    rows = cache[[3, 1, 0, 4, 2]].double().cpu().view(5, 2, nkv, ps, hd).permute(1, 0, 3, 2, 4).reshape(2, 5 * ps, nkv, hd)[:, :T]
    f64 = lambda v: v.double().cpu()      # noqa: E731
    want = P.mixed_head_attention(f64(q).view(T, nh, hd), rows[0], rows[1], hd ** -0.5, f64(r), f64(r), f64(talk), 10 ** 9)
    # the mixed weights (of both signs) and the result are rounded to bfloat16 (2^-9 each)
    assert rel_err(out[0], want.reshape(T, -1)) < 2e-2


@pytest.mark.parametrize("d,vd,heads,lens", [(128, 256, 2, (5, 15, 16, 50, 80)), (100, 30, 2, (33,)), (64, 63, 1, (48, 17)), (40, 5, 2, (47,))])
def test_mlstm_of_portions_in_two_roles(K, d, vd, heads, lens):
    torch.manual_seed(d + vd)
    T, W = sum(lens), vd + 1
    proj = torch.randn(T, heads * (2 * d + vd + 2), device="cuda")
    ib, fb, cap, g0 = torch.randn(heads, device="cuda"), torch.randn(heads, device="cuda") + 2, 15.0, heads * (2 * d + vd)
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    state = torch.randn(len(lens), heads * d * W + heads, device="cuda")
    S = state[:, :heads * d * W].double().cpu().view(-1, heads, d, W).clone()
    m = state[:, heads * d * W:].double().cpu().clone()
    f = proj.double().cpu()
    q, k = f[:, :heads * d].view(T, heads, d) * d ** -0.5, f[:, heads * d:2 * heads * d].view(T, heads, d)
    v = torch.cat([f[:, 2 * heads * d:g0].view(T, heads, vd), torch.ones(T, heads, 1, dtype=torch.float64)], 2)
    gi = cap * torch.tanh((f[:, g0:g0 + heads] + ib.double().cpu()) / cap)
    gf = torch.nn.functional.logsigmoid(cap * torch.tanh((f[:, g0 + heads:] + fb.double().cpu()) / cap))
    raw, top = torch.empty(T, heads, W, dtype=torch.float64), torch.empty(T, heads, dtype=torch.float64)
    for s in range(len(lens)):
        for t in range(cu[s], cu[s + 1]):
            new = torch.maximum(gf[t] + m[s], gi[t])
            S[s] = torch.exp(gf[t] + m[s] - new)[:, None, None] * S[s] + torch.exp(gi[t] - new)[:, None, None] * k[t][:, :, None] * v[t][:, None, :]
            m[s], top[t], raw[t] = new, new, torch.einsum("hdv,hd->hv", S[s], q[t])
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")      # noqa: E731
    got, got_top = K.mlstm_scan(proj, g0, g0 + heads, ib, fb, i32(cu), i32(list(range(len(lens)))), state, heads, d, vd, cap, max_q_len=max(lens))
    # float sums of d products; the gates' logarithms and exponentials to a few last places
    assert rel_err(got, raw.view(T, -1)) < 3e-6 and rel_err(got_top, top) < 1e-6 and rel_err(state[:, :heads * d * W], S.view(len(lens), -1)) < 3e-6


@pytest.mark.parametrize("d,vd,heads,lens", [(128, 256, 2, (1, 40, 16, 1)), (100, 30, 2, (33, 31, 2)), (64, 63, 1, (1,) * 26 + (130,)), (40, 5, 2, (47, 1)),
                                             (24, 6, 2, (1, 40)), (160, 6, 1, (2, 35))])
def test_mlstm_bits_do_not_depend_on_the_step(K, d, vd, heads, lens):
    """A request's outputs, maxima and state are the same bits alone, beside others and whichever kernels the steps take; a
    padding row (slot -1) leaves no state."""
    torch.manual_seed(d + vd)
    T, W, g0 = sum(lens), vd + 1, heads * (2 * d + vd)
    proj, ib, fb = torch.randn(T, g0 + 2 * heads, device="cuda"), torch.randn(heads, device="cuda"), torch.randn(heads, device="cuda") + 2
    before = torch.randn(len(lens), heads * d * W + heads, device="cuda")
    cu = torch.tensor((0,) + lens).cumsum(0).tolist()
    slots = list(range(len(lens)))
    if len(lens) > 2:
        slots[2] = -1
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")      # noqa: E731

    def run(a, b, cu, slots, state, longest):
        raw, top = K.mlstm_scan(proj[a:b].contiguous(), g0, g0 + heads, ib, fb, i32(cu), i32(slots), state, heads, d, vd, 15.0, max_q_len=longest)
        return [torch.cat([raw[cu[i]:cu[i + 1]], top[cu[i]:cu[i + 1]]], 1) for i in range(len(slots)) if slots[i] >= 0], state
    whole, state = run(0, T, cu, slots, before.clone(), max(lens))
    for longest in (1, T, None):
        y, s = run(0, T, cu, slots, before.clone(), longest)
        assert all(map(torch.equal, y, whole)) and torch.equal(s, state)
    assert len(lens) == 2 or torch.equal(state[2], before[2])
    for i, y in zip([i for i in range(len(lens)) if slots[i] >= 0], whole):
        got, s = run(cu[i], cu[i + 1], [0, lens[i]], [i], before.clone(), lens[i])
        assert torch.equal(got[0], y) and torch.equal(s[i], state[i])


@pytest.mark.parametrize("vocab,ctas", [(1000, 1), (2048, 2), (2049, 1), (40001, 4), (128256, 8)])
def test_top_p_rows_by_their_candidates(K, vocab, ctas):
    """Top-p alone: rows whose candidates reach the mass, fall short of it (flat: told by the bins' edges, or only by the candidates'
    masses), number just the limit, or hold infinities, draw what the general search over the whole row draws."""
    from ctypes import c_int
    torch.manual_seed(vocab)
    spread = [0.0, 0.01, 0.5, 1.0, 2.0, 4.0, 8.0, 100.0] * 3
    x = torch.randn(len(spread), vocab) * torch.tensor(spread)[:, None]
    x[3, ::2] = float("-inf")
    x[4, 7] = float("nan")
    x[5, vocab - 2] = float("inf")
    args = (x.cuda(), torch.full((24,), 0.9).cuda(), None, torch.tensor([0.9, 0.999, 1e-5] * 8).cuda(), torch.arange(24).cuda(), torch.arange(24).cuda() * 3)
    lib = K._lib("sampling.cu")
    try:
        lib.rv_sample_set_cluster(c_int(ctas))
        assert lib.rv_sample_set_short_way(c_int(0)) == 0
        general = K.sample(*args).tolist()
        assert lib.rv_sample_set_short_way(c_int(1)) == 0
        short = K.sample(*args).tolist()
        assert lib.rv_sample_set_short_way(c_int(2)) == 0
        served = K.sample(*args).tolist()                    # -1 where the short way hands the row on
    finally:
        lib.rv_sample_set_cluster(c_int(0)), lib.rv_sample_set_short_way(c_int(1))
    assert short[5] == vocab - 2
    # masses are added in different orders: a draw within rounding (2^-24 log2(vocab)) of a step may differ, one row in thousands
    rows = [r for r in range(24) if r != 5]
    assert sum(short[r] != general[r] for r in rows) <= 1
    # peaked rows go the short way (all but a thousandth of a wide row's mass may need more tokens than it holds); a flat row whose
    # tokens are more than it holds does not
    assert all(served[r] == short[r] for r in rows if spread[r] >= 4 and (r % 3 != 1 or vocab <= 2048))
    assert all(served[r] in (-1, short[r]) for r in rows)
    assert all((served[r] == -1) == (vocab > 2048) for r in (0, 16))


@pytest.mark.parametrize("temperature", [1e-30, 1e-39, 1e-42])
@pytest.mark.parametrize("k,p", [(0, 0.9), (50, 1.0), (50, 0.5), (0, 1.0)])
def test_temperatures_whose_reciprocal_overflows(K, temperature, k, p):
    """Ever lower temperatures draw the maximum, also where 1 / T is beyond the largest float; one of them where it is there twice."""
    torch.manual_seed(2)
    x = torch.randn(4, 5000, device="cuda")
    x[3, 7] = x[3, 9] = x[3].max() + 1
    full = lambda v, dtype: torch.full((4,), v, dtype=dtype, device="cuda")      # noqa: E731
    got = K.sample(x, full(temperature, torch.float32), full(k, torch.int32) if k else None, full(p, torch.float32) if p < 1 else None,
                   torch.arange(4, device="cuda"), torch.arange(4, device="cuda")).tolist()
    assert got[:3] == x[:3].argmax(1).tolist() and got[3] in (7, 9)


@pytest.mark.parametrize("T,nh,nkv,hd,dtype", [(3, 4, 2, 64, torch.bfloat16), (300, 6, 3, 20, torch.float32), (17, 32, 8, 128, torch.bfloat16), (1, 1, 1, 4, torch.float32)])
def test_row_kernels_in_words_of_four(K, T, nh, nkv, hd, dtype):
    """Rows on 16-byte boundaries are read in words of four elements by several blocks, rows at odd addresses one by one: the same
    bits where elements are copied, else the same to a few 2^-24 (or a rounding to bfloat16)."""
    torch.manual_seed(T + hd)
    rnd = lambda *shape: torch.randn(*shape, device="cuda")      # noqa: E731
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")      # noqa: E731

    def odd(t):
        return torch.empty(t.numel() + 1, dtype=t.dtype, device="cuda")[1:].view(t.shape).copy_(t)
    cols = nh * hd
    near = lambda a, b, tol=2e-6: rel_err(a, b.double().cpu()) < (tol if a.dtype == torch.float32 else 8e-3)      # noqa: E731
    x, e, v = rnd(T, cols), rnd(T, cols), rnd(2, cols).to(dtype)
    assert near(K.stream_add(x.clone(), e, v, 1), K.stream_add(odd(x), e, v, 1))
    assert near(K.scaled_sum(x.clone(), 0.5, e, 2.0), K.scaled_sum(odd(x), 0.5, e, 2.0))
    pair = rnd(T, 2 * cols)
    assert near(K.act_mul(pair, "swiglu_clamp", dtype, limit=1.5, alpha=1.7), K.act_mul(odd(pair), "swiglu_clamp", dtype, limit=1.5, alpha=1.7))
    alpha, w, b = rnd(1), rnd(cols), rnd(cols)
    assert near(K.dynamic_tanh(x, alpha, w, b, dtype), K.dynamic_tanh(odd(x), alpha, w, b, dtype))
    z = rnd(T, cols + 4).to(dtype)
    assert near(K.gated_group_rmsnorm(x, z, w, 1e-5, nh, dtype), K.gated_group_rmsnorm(odd(x), z, w, 1e-5, nh, dtype))
    pages, ps = -(-T // 8) + 1, 8
    slots, pos = i32([-1 if t == 2 else t + 3 for t in range(T)]), i32([(5 * t) % 40 for t in range(T)])
    ang = torch.rand(40, hd // 8 * 2, device="cuda") if hd >= 8 else None
    cos, sin = (ang.cos(), ang.sin()) if hd >= 8 else (None, None)
    proj = rnd(T, (nh + nkv) * hd)
    gq, gk = rnd(nh * hd).to(dtype), rnd(nkv * hd).to(dtype)
    out = []
    for p in (proj, odd(proj)):
        cache = torch.zeros(pages, 2, nkv, ps, hd, dtype=dtype, device="cuda")
        out.append((K.qk_norm_rope_cache_write(p, gq, gk, 1e-5, pos, cos, sin, slots, cache, nh, nkv, hd, dtype)[0], cache))
    assert all(near(a, b) for a, b in zip(*out))
    proj, out = rnd(T, (nh + 2 * nkv) * hd).to(dtype), []
    for p in (proj, odd(proj)):
        cache = torch.zeros(pages, nkv * ps * 2 * hd, dtype=dtype, device="cuda")
        out.append((K.kv_prepare(p, slots, cache, nh, nkv, hd, hd, 1e-6, dtype), cache))
    assert torch.equal(out[0][0], out[1][0]) and near(out[0][1], out[1][1])
    rot, rank = max(4, hd // 8 * 4), 12
    ang = torch.rand(40, rot // 2, device="cuda")
    proj, out = rnd(T, nh * (hd + rot) + rank + rot), []
    for p in (proj, odd(proj)):
        cache = torch.zeros(pages, 1, 1, ps, rank + rot, dtype=dtype, device="cuda")
        plain, row, _ = K.latent_prepare(p, w[:rank].contiguous() if cols >= rank else rnd(rank).fill_(0.7), 1e-5, pos, ang.cos(), ang.sin(), slots, cache, nh, hd, rot, rank,
                                         dtype, with_gate=False)
        out.append((plain, row[:, :, rank:], cache))
    assert torch.equal(out[0][0], out[1][0]) and near(out[0][1], out[1][1]) and near(out[0][2], out[1][2])
    for halves in (False, True):
        q = proj[:, :nh * (hd + rot)].contiguous()
        a, b = (K.latent_queries(p, pos, ang.cos(), ang.sin(), nh, hd, rot, rank, dtype, halves=halves) for p in (q, odd(q)))
        assert torch.equal(a[0], b[0]) and near(a[1][:, :, rank:], b[1][:, :, rank:])
