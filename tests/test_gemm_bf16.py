"""The tcgen05 matrix product alone, against float64, over both orientations, split
reductions, the SwiGLU epilogue, float32 output and ragged sizes."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def ops():
    from helios_b200.csrc import ops as _ops
    return _ops


def _case(T, N, K, seed, glu=False):
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(T, K, generator=g).to(torch.bfloat16)
    w = (torch.randn((2 * N if glu else N), K, generator=g) / K ** 0.5).to(torch.bfloat16)
    b = torch.randn(N, generator=g)
    return x, w, b


def _gated(gate, up, kind):
    act = gate * torch.sigmoid(gate) if kind in (True, "silu") else torch.nn.functional.gelu(gate, approximate="tanh")
    return act * up


def _close(got, want, scale=1.0):
    torch.testing.assert_close(got.double().cpu(), want, atol=2e-2 * scale, rtol=2e-2)


@pytest.mark.parametrize("T", [1, 8, 16, 17, 40, 64, 100, 128, 129, 300, 1000])
@pytest.mark.parametrize("N,K", [(128, 64), (200, 72), (384, 4096), (1000, 520), (4096, 1024)])
def test_plain_and_bias(T, N, K):
    x, w, b = _case(T, N, K, T + N)
    want = x.double() @ w.double().T
    _close(ops().linear_bf16(x.to(DEV), w.to(DEV)), want)
    _close(ops().linear_bf16(x.to(DEV), w.to(DEV), b.to(DEV)), want + b.double())
    got32 = ops().linear_bf16(x.to(DEV), w.to(DEV), out_dtype=torch.float32)
    assert got32.dtype == torch.float32
    torch.testing.assert_close(got32.double().cpu(), want, atol=2e-3, rtol=1e-3)
    ops().check_kernel_errors()


@pytest.mark.parametrize("cluster", [False, True])
@pytest.mark.parametrize("bn", [0, 16, 32, 64, 128])
@pytest.mark.parametrize("splits", [1, 2, 5, 8])
@pytest.mark.parametrize("glu", [False, "silu", "gelu_tanh"])
def test_every_orientation_and_split(bn, splits, glu, cluster):
    """Split reductions both ways: through scratch memory with a ticket per tile, and
    inside a thread-block cluster through distributed shared memory."""
    T = {0: 260, 16: 9, 32: 32, 64: 50, 128: 128}[bn]
    N, K = 392, 1024 + 64 * 3
    x, w, b = _case(T, N, K, bn + splits, glu)
    xd, wd = x.double(), w.double()
    if glu:
        gate, up = xd @ wd[:N].T, xd @ wd[N:].T
        want = _gated(gate, up, glu)
        got = ops().linear_bf16(x.to(DEV), w.to(DEV), glu=glu, plan=(bn, splits), cluster=cluster)
    else:
        want = xd @ wd.T + b.double()
        got = ops().linear_bf16(x.to(DEV), w.to(DEV), b.to(DEV), plan=(bn, splits), cluster=cluster)
    _close(got, want)
    ops().check_kernel_errors()


def test_split_sum_is_the_same_every_time_and_tickets_return_to_zero():
    x, w, _ = _case(8, 4096, 14336, 3)
    xd, wd = x.to(DEV), w.to(DEV)
    first = ops().linear_bf16(xd, wd, plan=(16, 7), cluster=False)
    for _ in range(5):
        assert torch.equal(ops().linear_bf16(xd, wd, plan=(16, 7), cluster=False), first)
    # the cluster reduction adds the slices in the same order
    for _ in range(3):
        assert torch.equal(ops().linear_bf16(xd, wd, plan=(16, 7), cluster=True), first)
    _, tickets, _ = ops()._gemm_workspace(torch.device(DEV))
    assert int(tickets.abs().sum()) == 0
    _close(first, x.double() @ w.double().T)
    ops().check_kernel_errors()


@pytest.mark.parametrize("T", [3, 64, 2048])
def test_model_sized_products(T):
    # the shapes of the 8B model's layer: fused QKV, output, gate/up with SwiGLU, down
    for N, K, glu in [(6144, 4096, False), (4096, 4096, False), (14336, 4096, True), (4096, 14336, False)]:
        x, w, _ = _case(T, N, K, T + N, glu)
        xd, wd = x.double(), w.double()
        if glu:
            gate, up = xd @ wd[:N].T, xd @ wd[N:].T
            want = gate * torch.sigmoid(gate) * up
            got = ops().linear_swiglu(x.to(DEV), w.to(DEV))
        else:
            want = xd @ wd.T
            got = ops().linear(x.to(DEV), w.to(DEV))
        _close(got, want)
    ops().check_kernel_errors()


def test_k_that_is_no_multiple_of_8_goes_to_the_library_and_is_refused_by_the_kernel():
    x, w, _ = _case(5, 64, 100, 1)
    got = ops().linear(x.to(DEV), w.to(DEV))
    _close(got, x.double() @ w.double().T)
    with pytest.raises(ops().KernelError):
        ops().linear_bf16(x.to(DEV), w.to(DEV))


@pytest.mark.parametrize("two_sm", [False, True])
@pytest.mark.parametrize("T,N,K", [(129, 256, 64), (256, 512, 192), (300, 392, 1224), (2048, 4096, 1024),
                                   (1000, 1000, 520), (513, 6144, 4096)])
@pytest.mark.parametrize("glu", [False, "silu", "gelu_tanh"])
def test_prefill_kernels_one_and_two_sm(T, N, K, glu, two_sm):
    """Tokens on the M axis: one block per 128x256 tile, and the persistent cta_group::2
    kernel (pairs of SMs on 256x256 tiles), ragged in every dimension."""
    x, w, b = _case(T, N, K, T + N + K, glu)
    xd, wd = x.double(), w.double()
    if glu:
        gate, up = xd @ wd[:N].T, xd @ wd[N:].T
        want = _gated(gate, up, glu)
        got = ops().linear_bf16(x.to(DEV), w.to(DEV), glu=glu, plan=(0, 1), two_sm=two_sm)
    else:
        want = xd @ wd.T + b.double()
        got = ops().linear_bf16(x.to(DEV), w.to(DEV), b.to(DEV), plan=(0, 1), two_sm=two_sm)
    ops().check_kernel_errors()
    _close(got, want)
    got32 = ops().linear_bf16(x.to(DEV), w.to(DEV), glu=glu, plan=(0, 1), two_sm=two_sm, out_dtype=torch.float32)
    ops().check_kernel_errors()
    assert got32.dtype == torch.float32


# ------------------------------------------------------------------ the epilogues of few-token steps
def _norm_case(T, N, K, seed):
    g = torch.Generator().manual_seed(seed)
    x, w, b = _case(T, N, K, seed)
    residual = torch.randn(T, N, generator=g) * 3.0
    residual[:, 5 % N] *= 40.0                       # one feature far larger than the rest
    norm_w = 1.0 + 0.3 * torch.randn(N, generator=g)
    return x, w, b, residual, norm_w


@pytest.mark.parametrize("way", ["cluster", "scratch", "whole"])
@pytest.mark.parametrize("T", [1, 8, 16, 17, 32])
@pytest.mark.parametrize("N,K", [(4096, 4096), (896, 4864), (200, 72), (384, 14336)])
def test_a_product_into_the_residual_leaves_the_next_norms_input(T, N, K, way):
    """residual += x W^T (+ bias); out = bfloat16(residual * norm weight); the partial sums of
    squares add up to sum(residual^2): every way the reduction can be split."""
    x, w, b, residual, norm_w = _norm_case(T, N, K, T * 7 + N + K)
    bn = 16 if T <= 16 else 32
    # 2 and 3 slices hold 64 and 43 of a tile's 128 features each (two rows a lane), 5 hold 26
    splits = 1 if way == "whole" else min(2 + (T + N) % 4, max(1, (K // 64) // 2))
    res = residual.to(DEV).clone()
    got = ops().linear_bf16(x.to(DEV), w.to(DEV), b.to(DEV), plan=(bn, splits), cluster=(way == "cluster"),
                            residual=res, norm_weight=norm_w.to(DEV))
    scaled, sumsq = got
    want_res = residual.double() + x.double() @ w.double().T + b.double()
    torch.testing.assert_close(res.double().cpu(), want_res, atol=2e-3, rtol=1e-3)
    assert scaled.dtype == torch.bfloat16 and tuple(sumsq.shape) == (T, 8 * -(-N // 128))
    # bit-equal to rounding what the kernel itself left in the residual
    assert torch.equal(scaled.cpu(), (res.cpu() * norm_w).to(torch.bfloat16))
    torch.testing.assert_close(sumsq.double().sum(1).cpu(), (res.double().cpu() ** 2).sum(1), rtol=1e-5, atol=0)
    # without a norm weight only the residual moves
    res2 = residual.to(DEV).clone()
    assert ops().linear_bf16(x.to(DEV), w.to(DEV), plan=(bn, splits), cluster=(way == "cluster"),
                             residual=res2) is None
    torch.testing.assert_close(res2.double().cpu(), want_res - b.double(), atol=2e-3, rtol=1e-3)
    ops().check_kernel_errors()


@pytest.mark.parametrize("way", ["cluster", "scratch", "whole"])
@pytest.mark.parametrize("glu", [False, True])
@pytest.mark.parametrize("T", [1, 8, 17, 32])
@pytest.mark.parametrize("N,K", [(6144, 4096), (1152, 896), (200, 72)])
def test_a_product_applies_the_tokens_rms_factor(T, N, K, glu, way):
    """Input rows that lack 1 / rms: the accumulators get it before bias or SwiGLU."""
    x, w, b = _case(T, N, K, T + N + K, glu)
    g = torch.Generator().manual_seed(T)
    slots = 8 * -(-K // 128)
    sumsq = torch.rand(T, slots, generator=g) * (K / slots) * torch.linspace(0.1, 30.0, T)[:, None]
    eps = 1e-5
    rstd = torch.rsqrt(sumsq.double().sum(1) / K + eps)[:, None]
    bn = 16 if T <= 16 else 32
    splits = 1 if way == "whole" else min(5, max(1, (K // 64) // 2))
    kw = dict(plan=(bn, splits), cluster=(way == "cluster"), sumsq=sumsq.to(DEV), eps=eps)
    xd, wd = x.double(), w.double()
    if glu:
        gate, up = rstd * (xd @ wd[:N].T), rstd * (xd @ wd[N:].T)
        want = gate * torch.sigmoid(gate) * up
        got = ops().linear_bf16(x.to(DEV), w.to(DEV), glu=True, **kw)
    else:
        want = rstd * (xd @ wd.T) + b.double()
        got = ops().linear_bf16(x.to(DEV), w.to(DEV), b.to(DEV), **kw)
    _close(got, want, scale=float(want.abs().max().clamp(min=1.0)) / 4)
    ops().check_kernel_errors()


def test_two_products_with_the_norm_between_them_folded_in():
    """O-projection into the residual, then gate|up with the token factors: the same as
    add, RMSNorm and the product one after the other."""
    T, H, I = 8, 4096, 1024
    x, wo, _b, residual, norm_w = _norm_case(T, H, H, 99)
    g = torch.Generator().manual_seed(5)
    wgu = (torch.randn(2 * I, H, generator=g) / H ** 0.5).to(torch.bfloat16)
    eps = 1e-5
    res = residual.to(DEV).clone()
    scaled, sumsq = ops().linear_bf16(x.to(DEV), wo.to(DEV), residual=res, norm_weight=norm_w.to(DEV))
    got = ops().linear_bf16(scaled, wgu.to(DEV), glu=True, sumsq=sumsq, eps=eps)
    new = residual.double() + x.double() @ wo.double().T
    normed = new * torch.rsqrt((new ** 2).mean(1, keepdim=True) + eps) * norm_w.double()
    gate, up = normed @ wgu.double()[:I].T, normed @ wgu.double()[I:].T
    _close(got, gate * torch.sigmoid(gate) * up, scale=2.0)
    assert ops().DEFERRED_NORM_TOKENS <= ops().DEFERRED_NORM_MOST == 32
    with pytest.raises(ops().KernelError):
        ops().linear_bf16(torch.zeros(40, H, dtype=torch.bfloat16, device=DEV), wo.to(DEV),
                          residual=torch.zeros(40, H, device=DEV))
    ops().check_kernel_errors()


@pytest.mark.parametrize("T", [129, 255, 257])
@pytest.mark.parametrize("N", [16, 250, 252, 255, 256, 260, 1001])
def test_float32_output_of_the_two_sm_kernel_at_odd_widths(T, N):
    """Rows that are and are not whole 16-byte pieces, and a last piece of sixteen columns that is cut."""
    x, w, _b = _case(T, N, 136, T * N)
    got = ops().linear_bf16(x.to(DEV), w.to(DEV), plan=(0, 1), two_sm=True, out_dtype=torch.float32)
    torch.testing.assert_close(got.double().cpu(), x.double() @ w.double().T, atol=2e-3, rtol=1e-3)


@pytest.mark.parametrize("T", [1, 2, 3, 4])
@pytest.mark.parametrize("N,K", [(16, 8), (100, 248), (129, 256), (896, 264), (1152, 896), (17, 2048), (250, 2056), (896, 4864)])
def test_products_of_few_tokens_with_a_small_weight(T, N, K, monkeypatch):
    """Every epilogue of the kernel on the FMA pipes against float64: one and two warps a row, rows that
    end inside a step of 256, features that end inside a block and inside a slot of the squares."""
    o = ops()
    monkeypatch.setattr(o, "GEMV_WEIGHT_BYTES", {1: 1 << 30, 2: 1 << 30, 3: 1 << 30, 4: 1 << 30})
    x, w, b = _case(T, N, K, T + N + K)
    xd, wd, bd = x.to(DEV), w.to(DEV), b.to(DEV)
    want = x.double() @ w.double().T
    _close(o.linear_bf16(xd, wd), want)
    _close(o.linear_bf16(xd, wd, bd), want + b.double())
    # float32 out: K products, each sum of 8 * K / 256 + 6 roundings
    bound = (K / 32 + 8) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T) + 1e-6
    assert ((o.linear_bf16(xd, wd, out_dtype=torch.float32).double().cpu() - want).abs() <= bound).all()
    g = torch.Generator().manual_seed(K)
    slots = torch.rand(T, 8 * -(-K // 128), generator=g)
    inv = torch.rsqrt(slots.double().sum(-1, keepdim=True) / K + 1e-5)
    _close(o.linear_bf16(xd, wd, bd, sumsq=slots.to(DEV), eps=1e-5), want * inv + b.double(), scale=float(inv.max()) + 1)
    res, nw = torch.randn(T, N, generator=g), torch.rand(N, generator=g) + 0.5
    r1 = res.to(DEV)
    assert o.linear_bf16(xd, wd, residual=r1) is None
    assert ((r1.double().cpu() - res.double() - want).abs() <= bound + 1e-6).all()
    r2 = res.to(DEV)
    scaled, squares = o.linear_bf16(xd, wd, bd, residual=r2, norm_weight=nw.to(DEV))
    assert ((r2.double().cpu() - res.double() - want - b.double()).abs() <= bound + 1e-6).all()
    assert torch.equal(scaled.cpu(), (r2.cpu() * nw).to(torch.bfloat16))
    torch.testing.assert_close(squares.double().cpu().sum(-1), (r2.double().cpu() ** 2).sum(-1), rtol=1e-5, atol=1e-6)
    # the same through the tensor-core kernel, and a row alone is the row in the batch
    first = o.linear_bf16(xd, wd, out_dtype=torch.float32)
    assert torch.equal(o.linear_bf16(xd[T - 1:].contiguous(), wd, out_dtype=torch.float32), first[T - 1:])
    monkeypatch.setattr(o, "GEMV_WEIGHT_BYTES", {})
    torch.testing.assert_close(o.linear_bf16(xd, wd, out_dtype=torch.float32), first, atol=2e-4, rtol=1e-4)


@pytest.mark.parametrize("kind", ["silu", "gelu_tanh"])
@pytest.mark.parametrize("N,K", [(16, 8), (100, 248), (129, 256), (4864, 896), (17, 2048), (250, 2056), (64, 4864)])
def test_gated_units_of_one_token_with_a_small_weight(N, K, kind):
    """As above, with and without the token's 1 / rms; gate and up rows of a feature end together."""
    o = ops()
    assert 2 * N * K * 2 <= o.GEMV_GATED_WEIGHT_BYTES
    x, w, _b = _case(1, N, K, N + K, glu=True)
    both = x.double() @ w.double().T
    _close(o.linear_bf16(x.to(DEV), w.to(DEV), glu=kind), _gated(both[:, :N], both[:, N:], kind))
    slots = torch.rand(1, 8 * -(-K // 128), generator=torch.Generator().manual_seed(K))
    both = both * torch.rsqrt(slots.double().sum(-1, keepdim=True) / K + 1e-5)
    got = o.linear_bf16(x.to(DEV), w.to(DEV), glu=kind, sumsq=slots.to(DEV), eps=1e-5).double().cpu()
    # one rounding to eight bits, after sums of 32 bits
    torch.testing.assert_close(got, _gated(both[:, :N], both[:, N:], kind), rtol=2.0 ** -8, atol=1e-4)


@pytest.mark.parametrize("cluster", [0, 2])
@pytest.mark.parametrize("out_dtype,offset", [(torch.float32, 0), (torch.float32, 1), (torch.float32, 2), (torch.bfloat16, 0),
                                              (torch.bfloat16, 1), (torch.bfloat16, 4)])
def test_results_at_addresses_that_are_no_whole_pieces(out_dtype, offset, cluster):
    """The exported function takes any address for its results (the Python call allocates them): the kernels
    for many tokens, one and two SMs a tile, store value by value where 16-byte stores would be misaligned."""
    import ctypes

    o = ops()
    T, N, K = 257, 272, 136
    x, w, _b = _case(T, N, K, offset)
    xd, wd = x.to(DEV), w.to(DEV)
    o.linear_bf16(xd, wd)                                     # (sets the function's argument types)
    _scratch, _tickets, err = o._gemm_workspace(xd.device)
    room = torch.full((T * N + 8 + offset,), 7.0, dtype=out_dtype, device=DEV)
    out = room[offset:offset + T * N]
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    f = o.load_library("gemm_bf16").hb_gemm_bf16
    rc = f(p(out), p(xd), p(wd), None, None, None, p(err), T, N, K, K, K, N, N, 0, 0, int(out_dtype == torch.float32), 0, 1,
           cluster, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    torch.cuda.synchronize()
    want = x.double() @ w.double().T
    if out_dtype == torch.float32:
        torch.testing.assert_close(out.view(T, N).double().cpu(), want, atol=2e-3, rtol=1e-3)
    else:
        _close(out.view(T, N), want)
    assert bool((room[offset + T * N:] == 7).all()) and bool((room[:offset] == 7).all())


@pytest.mark.parametrize("settings", [dict(cluster=True), dict(cluster=False), dict(two_sm=False), dict(plan=(16, 1)), {}])
@pytest.mark.parametrize("glu", [False, True])
def test_settings_of_the_tensor_core_kernels_choose_them(settings, glu, monkeypatch):
    """One token and a small weight, which go to the FMA pipes unless the caller sets something of the others."""
    o, seen = ops(), []
    plain = o._fn
    monkeypatch.setattr(o, "_fn", lambda lib, name, types: seen.append(name) or plain(lib, name, types))
    x, w, _b = _case(1, 256, 512, 5, glu=glu)
    got = o.linear_bf16(x.to(DEV), w.to(DEV), glu=glu, **settings)
    want = x.double() @ w.double().T
    _close(got, _gated(want[:, :256], want[:, 256:], True) if glu else want)
    assert seen == ["hb_gemm_bf16" if settings else "hb_gemv_bf16"]


@pytest.mark.parametrize("T,N,K,gated,takes", [
    (1, 16 * 296, 2048, False, True), (1, 16 * 296 + 1, 2048, False, False), (1, 16 * 333, 1024, False, True),
    (1, 16 * 333 + 1, 1024, False, False), (1, 16 * 296 + 1, 248, False, False), (1, 16 * 333, 256, False, True), (1, 16 * 148, 2056, False, True),
    (1, 16 * 148 + 1, 2056, False, False), (1, 32000, 512, False, False), (1, 16, 65536, False, True),
    (2, 16 * 296, 1024, False, True), (2, 16 * 296 + 1, 1024, False, False), (2, 768, 1032, False, True), (2, 769, 2048, False, False),
    (2, 1024, 2056, False, True), (2, 1025, 2056, False, False), (2, 1024, 4096, False, True), (2, 16, 4104, False, False),
    (3, 1536, 1024, False, True), (4, 1537, 1024, False, False), (4, 16, 1032, False, False), (5, 16, 64, False, False),
    (1, 8288, 1024, True, True), (1, 8289, 1024, True, False), (1, 16 * 296, 1032, True, True), (1, 16 * 296 + 1, 1032, True, False),
    (1, 1024, 4864, True, True), (1, 1024, 4872, True, False), (1, 16 * 296, 2048, True, True), (2, 16, 64, True, False)])
def test_which_products_the_fma_pipes_take(T, N, K, gated, takes, monkeypatch):
    """By rounds of blocks of 16 features on 148 SMs and by the length of a row, at the edges."""
    o = ops()
    monkeypatch.setattr(o, "sm_count", lambda device=None: 148)
    assert o._on_fma_pipes(T, N, K, gated) == takes


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["silu", "gelu_tanh"])
@pytest.mark.parametrize("T,N,K", [(129, 40, 64), (256, 128, 72), (257, 200, 128), (700, 333, 512)])
def test_gated_unit_with_biases_in_the_epilogue(T, N, K, kind):
    """The two-SM kernel adds gate's and up's biases to its float32 sums; ragged rows and features."""
    g = torch.Generator().manual_seed(T + N)
    x, w = torch.randn(T, K, generator=g).bfloat16(), (torch.randn(2 * N, K, generator=g) * K ** -0.5).bfloat16()
    b = torch.randn(2 * N, generator=g)
    got = ops().linear_bf16(x.cuda(), w.cuda(), glu=kind, glu_bias=b.cuda()).cpu().double()
    y = x.double() @ w.double().T + b.double()
    act = torch.nn.functional.silu if kind == "silu" else (lambda t: torch.nn.functional.gelu(t, approximate="tanh"))
    want = act(y[:, :N]) * y[:, N:]
    # one rounding to eight bits, after sums of 32 bits
    assert ((got - want).abs() <= 2.0 ** -8 * want.abs() + 2e-5).all()
    with pytest.raises(ops().KernelError):
        ops().linear_bf16(x[:128].cuda(), w.cuda(), glu=kind, glu_bias=b.cuda())
    with pytest.raises(ops().KernelError):
        ops().linear_bf16(x.cuda(), w.cuda(), glu=kind, bias=b[:N].cuda())


@pytest.mark.gpu
@pytest.mark.parametrize("T", [1, 2, 4])
@pytest.mark.parametrize("N,K", [(1184, 520), (1185, 520), (2304, 1000), (2305, 1000), (1100, 2056), (1184, 512)])
def test_products_of_few_tokens_with_blocks_of_eight_and_sixteen_features(T, N, K, monkeypatch):
    """Both sides of the sizes at which blocks have eight features, and a partial sum of squares each;
    given tensors keep eight slots to 128 features."""
    o = ops()
    monkeypatch.setattr(o, "GEMV_WEIGHT_BYTES", {1: 1 << 30, 2: 1 << 30, 4: 1 << 30})
    g = torch.Generator().manual_seed(N + K)
    x, w = torch.randn(T, K, generator=g).bfloat16().cuda(), (torch.randn(N, K, generator=g) * K ** -0.5).bfloat16().cuda()
    res, nw = torch.randn(T, N, generator=g).cuda(), (torch.rand(N, generator=g) + 0.5).cuda()
    want = res.double() + x.double() @ w.double().T
    given = (torch.empty(T, N, dtype=torch.bfloat16, device="cuda"), torch.full((T, 8 * -(-N // 128)), float("nan"), device="cuda"))
    for out in (None, given):
        r = res.clone()
        scaled, squares = o.linear_bf16(x, w, residual=r, norm_weight=nw, norm_out=out)
        # float32 sums of K products of order 1 / K
        assert (r.double() - want).abs().max() < 1e-5
        assert torch.equal(scaled, (r * nw).bfloat16())
        torch.testing.assert_close(squares.double().sum(-1), (r.double() ** 2).sum(-1), rtol=1e-5, atol=1e-6)


@pytest.mark.gpu
@pytest.mark.parametrize("N", [4736, 4737, 5328, 5329, 5921])
def test_gated_units_of_one_token_with_blocks_of_eight_to_ten_warps(N):
    """Blocks of 16, 18 and 20 features, whichever need the fewest rounds."""
    o, K = ops(), 520
    g = torch.Generator().manual_seed(N)
    x, w = torch.randn(1, K, generator=g).bfloat16().cuda(), (torch.randn(2 * N, K, generator=g) * K ** -0.5).bfloat16().cuda()
    slots = torch.rand(1, 24, generator=g).cuda()
    y = (x.double() @ w.double().T) * torch.rsqrt(slots.double().sum() / K + 1e-5)
    want = torch.nn.functional.silu(y[:, :N]) * y[:, N:]
    got = o.linear_bf16(x, w, glu=True, sumsq=slots, eps=1e-5)
    assert ((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2e-4).all()
