"""The kernels of the recurrent mixers (causal convolution, selective scan, minimal gated recurrence, gated
delta rule) and the small kernels that go with them, each alone against its plain PyTorch version
(tests/ref_ops.py), in 32-bit and in bfloat16: spans of several lengths beside single tokens, a second
step that continues from the state the first one left, a step of single tokens only, empty spans, sizes
that are no power of two and no multiple of a warp."""
import pytest
import torch

import ref_ops
from test_gpu_kernels import make_step

pytestmark = pytest.mark.gpu

DTYPES = [torch.float32, torch.bfloat16]
# the last two are long enough for the passes over chunks of rows (chunks that end inside and at a request's end,
# a request shorter than a chunk, one of exactly two chunks)
STEPS = ([1, 3, 4, 11, 1], [5, 1, 1, 2, 9], [1, 1, 1, 1, 1], [2, 37, 1, 1, 6], [200, 1, 63, 128, 70], [64, 65, 300, 2, 1])
MANY_SINGLES = [1] * 20           # more single tokens than the one-kernel paths for few requests take


def ops():
    from zig_ai_b200.kernels import ops as o
    o.require(extra=("causal_conv", "selective_scan", "min_gru", "gated_delta"))
    return o


def tol(dtype):
    return dict(atol=3e-5, rtol=3e-5) if dtype == torch.float32 else dict(atol=3e-2, rtol=3e-2)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("C,L,bias,act", [(96, 4, True, True), (64, 3, False, True), (200, 2, True, False), (48, 1, False, True),
                                          (130, 7, True, True)])
def test_causal_conv_spans_and_state(dtype, C, L, bias, act):
    o = ops()
    g = torch.Generator().manual_seed(4)
    w = (torch.randn(C, L, generator=g) * 0.3).cuda()
    b = (torch.randn(C, generator=g) * 0.3).cuda() if bias else None
    state_a = torch.randn(6, max(L - 1, 1), C, generator=g).cuda()
    state_b = state_a.clone()
    for q_lens in STEPS:
        step = make_step(o, dtype, [3] * 5, q_lens, 8, 256, 5)
        wide = torch.randn(sum(q_lens), C + 24, generator=g).to(dtype).cuda()
        x = wide[:, 8:8 + C]                                   # a column slice of a wider matrix
        ya = o.causal_conv(x, w, b, state_a, step, act, True)
        yb = ref_ops.causal_conv(x, w, b, state_b, step, act, True)
        assert torch.allclose(ya.float(), yb.float(), **tol(dtype)), q_lens
        assert torch.allclose(state_a, state_b, atol=1e-6, rtol=1e-6), q_lens
    keep = state_a.clone()
    step = make_step(o, dtype, [3] * 5, [2, 4, 1, 1, 3], 8, 64, 5)
    x = torch.randn(11, C, generator=g).to(dtype).cuda()
    o.causal_conv(x, w, b, state_a, step, act, False)          # write_state off: the history stays
    assert torch.equal(state_a, keep)
    assert torch.equal(state_a[0], state_b[0])                 # the null slot was never touched


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("I,S,R", [(96, 20, 12), (70, 3, 5), (33, 16, 1), (40, 40, 7), (20, 100, 9), (12, 200, 3)])
def test_selective_scan(dtype, I, S, R):
    o = ops()
    g = torch.Generator().manual_seed(6)
    w_dt = (torch.randn(I, R, generator=g) * 0.5).to(dtype).cuda()
    b_dt = (torch.randn(I, generator=g) * 0.5).cuda()
    a_log = (torch.randn(I, S, generator=g) * 0.5).cuda()
    d = torch.randn(I, generator=g).cuda()
    state_a = torch.randn(6, I, S, generator=g).cuda()
    state_b = state_a.clone()
    for q_lens in STEPS:
        step = make_step(o, dtype, [3] * 5, q_lens, 8, 256, 5)
        N = sum(q_lens)
        x = torch.randn(N, I, generator=g).to(dtype).cuda()
        proj = torch.randn(N, R + 2 * S + 3, generator=g).to(dtype).cuda()
        z = torch.randn(N, 2 * I, generator=g).to(dtype).cuda()[:, I:]
        ya = o.selective_scan(x, proj, z, w_dt, b_dt, a_log, d, state_a, step, R, True)
        yb = ref_ops.selective_scan(x, proj, z, w_dt, b_dt, a_log, d, state_b, step, R, True)
        assert torch.allclose(ya.float(), yb.float(), **tol(dtype)), q_lens
        assert torch.allclose(state_a, state_b, atol=1e-4, rtol=1e-4), q_lens
    assert torch.equal(state_a[0], state_b[0])


@pytest.mark.parametrize("dtype", DTYPES)
def test_selective_scan_single_tokens_aligned_rows(dtype):
    """A step of single tokens sums the step size's product itself, 16 bytes a load where the rows allow it."""
    o = ops()
    g = torch.Generator().manual_seed(13)
    I, S, R = 72, 16, 32
    w_dt = (torch.randn(I, R, generator=g) * 0.5).to(dtype).cuda()
    b_dt, a_log, d = (torch.randn(I, generator=g) * 0.5).cuda(), (torch.randn(I, S, generator=g) * 0.5).cuda(), torch.randn(I, generator=g).cuda()
    state_a = torch.randn(6, I, S, generator=g).cuda()
    state_b = state_a.clone()
    for _ in range(3):
        step = make_step(o, dtype, [3] * 5, [1] * 5, 8, 64, 5)
        x = torch.randn(5, I, generator=g).to(dtype).cuda()
        proj = torch.randn(5, R + 2 * S, generator=g).to(dtype).cuda()
        z = torch.randn(5, I, generator=g).to(dtype).cuda()
        ya = o.selective_scan(x, proj, z, w_dt, b_dt, a_log, d, state_a, step, R, True)
        yb = ref_ops.selective_scan(x, proj, z, w_dt, b_dt, a_log, d, state_b, step, R, True)
        assert torch.allclose(ya.float(), yb.float(), **tol(dtype))
        assert torch.allclose(state_a, state_b, atol=1e-4, rtol=1e-4)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("W", [200, 70, 1, 130])
def test_min_gru(dtype, W):
    o = ops()
    g = torch.Generator().manual_seed(7)
    bz, bx = torch.randn(W, generator=g).cuda(), torch.randn(W, generator=g).cuda()
    state_a = torch.randn(6, W, generator=g).cuda()
    state_b = state_a.clone()
    for q_lens in STEPS:
        step = make_step(o, dtype, [3] * 5, q_lens, 8, 256, 5)
        zxg = (torch.randn(sum(q_lens), 3 * W, generator=g) * 2).to(dtype).cuda()
        ya = o.min_gru(zxg, bz, bx, state_a, step, True)
        yb = ref_ops.min_gru(zxg, bz, bx, state_b, step, True)
        assert torch.allclose(ya.float(), yb.float(), **tol(dtype)), q_lens
        assert torch.allclose(state_a, state_b, atol=1e-5, rtol=1e-5), q_lens
    assert torch.equal(state_a[0], state_b[0])


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("H,G,D,V", [(6, 2, 32, 40), (2, 2, 16, 24), (3, 1, 40, 33), (4, 2, 64, 128), (2, 1, 128, 48),
                                     (1, 1, 200, 20), (2, 1, 8, 70)])
def test_gated_delta(dtype, H, G, D, V):
    o = ops()
    g = torch.Generator().manual_seed(8)
    a_log, dt_bias = torch.randn(H, generator=g).cuda() * 0.5, torch.randn(H, generator=g).cuda() * 0.5
    norm_w = (1 + 0.1 * torch.randn(V, generator=g)).cuda()
    state_a = (torch.randn(22, H, D, V, generator=g) * 0.3).cuda()
    state_b = state_a.clone()
    cols = 2 * G * D + H * V
    for q_lens in STEPS + (MANY_SINGLES,):
        step = make_step(o, dtype, [3] * len(q_lens), q_lens, 8, 256, 5)
        N = sum(q_lens)
        qkv = torch.randn(N, cols, generator=g).to(dtype).cuda()
        rest = torch.randn(N, H * V + 2 * H, generator=g).to(dtype).cuda()
        gate, b, a = rest[:, :H * V], rest[:, H * V:H * V + H], rest[:, H * V + H:]
        ya = o.gated_delta(qkv, b, a, gate, a_log, dt_bias, norm_w, 1e-5, state_a, step, H, G, D, V, True)
        yb = ref_ops.gated_delta(qkv, b, a, gate, a_log, dt_bias, norm_w, 1e-5, state_b, step, H, G, D, V, True)
        assert torch.allclose(ya.float(), yb.float(), **tol(dtype)), q_lens
        assert torch.allclose(state_a, state_b, atol=1e-4, rtol=1e-4), q_lens
    assert torch.equal(state_a[0], state_b[0])


@pytest.mark.parametrize("channel", [False, True])
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("singles,spans", [(8, [2]), (9, [70, 5]), (17, [64, 0, 63]), (32, [66]), (7, [130]), (8, [70]), (12, [64, 0, 130]),
                                           (16, [66]), (8, [0, 0]), (17, [64, 0])])
@pytest.mark.parametrize("captured", [False, True])
def test_gated_delta_of_decoded_tokens_ahead_of_spans(singles, spans, captured, dtype, channel):
    """Leading spans of one token (8 to 128) take the one kernel where every other span goes in chunks (rows and states are then those of
    a step of the same requests alone, to the bit, and the walk's kernels do not run); everything else is walked, and so is a step in
    the layout of a captured shape (empty spans, counts of chunks and spans rounded up)."""
    o = ops()
    g = torch.Generator().manual_seed(27)
    H, G, D, V = 4, 2, 64, 128
    q_lens = [1] * singles + spans + ([0, 0] if captured else [])
    N = sum(q_lens)
    step = make_step(o, dtype, [3] * len(q_lens), q_lens, 8, 256, 5)
    if captured:
        step.attn_tiles = N // 128 + len(q_lens)
    assert step.single_first == (singles if singles == 8 else 0 if singles < 8 else 1 << (singles.bit_length() - 1))
    qkv, b, a, gate, a_log, dt_bias, norm_w = (t.to(dtype) if t.dtype == torch.bfloat16 else t for t in delta_inputs(H, G, D, V, N, channel, g))
    state_a = (torch.randn(len(q_lens) + 3, H, D, V, generator=g) * 0.3).cuda()
    state_b, state_c = state_a.clone(), state_a.clone()
    before = o.launches
    ya = o.gated_delta(qkv, b, a, gate, a_log, dt_bias, norm_w, 1e-5, state_a, step, H, G, D, V, True, channel_decay=channel)
    launches = o.launches - before
    yb = ref_ops.gated_delta(qkv, b, a, gate, a_log, dt_bias, norm_w, 1e-5, state_b, step, H, G, D, V, True, channel_decay=channel)
    # the limits of test_gated_delta
    assert torch.allclose(ya.float(), yb.float(), **tol(dtype))
    assert torch.allclose(state_a, state_b, atol=1e-4, rtol=1e-4)
    chunked = dtype == torch.bfloat16
    if not captured and singles >= 8 and all(n == 0 or (n >= 64 and chunked) for n in spans):
        for i in range(0, singles, 16):                          # (steps of up to 16 single tokens are that kernel's)
            k = min(i + 16, singles)
            alone = make_step(o, dtype, [3] * (k - i), [1] * (k - i), 8, 256, 5, slots=list(range(i + 1, k + 1)))
            yc = o.gated_delta(*(t[i:k].contiguous() for t in (qkv, b, a, gate)), a_log, dt_bias, norm_w, 1e-5, state_c, alone, H, G, D, V, True,
                               channel_decay=channel)
            assert torch.equal(ya[i:k], yc)
        assert torch.equal(state_a[1:singles + 1], state_c[1:singles + 1])
        assert launches == 2 + (2 if any(spans) else 0)          # the one kernel, the chunks' two, the norm of their rows
    else:
        long = N >= 64 if captured else any(n >= 64 for n in spans)
        assert launches == 3 + (2 if long and chunked else 0)    # the walk's two, the chunks' two, the norm
    assert o.read_status() == 0


@pytest.mark.parametrize("dtype", DTYPES)
def test_empty_spans_change_nothing(dtype):
    """A step may hold spans without tokens (a captured step shape is filled up with them)."""
    o = ops()
    g = torch.Generator().manual_seed(9)
    step = make_step(o, dtype, [3, 0, 5], [4, 0, 2], 8, 64, 5)
    W = 40
    state = torch.randn(6, W, generator=g).cuda()
    before = state.clone()
    zxg = torch.randn(6, 3 * W, generator=g).to(dtype).cuda()
    o.min_gru(zxg, None, None, state, step, True)
    assert torch.equal(state[2], before[2]) and not torch.equal(state[1], before[1])
    conv_state = torch.randn(6, 3, W, generator=g).cuda()
    before = conv_state.clone()
    o.causal_conv(zxg[:, :W], torch.randn(W, 4, generator=g).cuda(), None, conv_state, step, True, True)
    assert torch.equal(conv_state[2], before[2]) and not torch.equal(conv_state[3], before[3])


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("kind", ["gelu", "gelu_tanh", "silu", "relu"])
@pytest.mark.parametrize("shape", [(3, 192), (7, 1001)])
def test_activation_and_weighted_sum(dtype, kind, shape):
    o = ops()
    g = torch.Generator().manual_seed(10)
    x = (torch.randn(*shape, generator=g) * 3).to(dtype).cuda()
    y = (torch.randn(*shape, generator=g) * 3).to(dtype).cuda()
    assert torch.allclose(o.activation(x, kind).float(), ref_ops.activation(x, kind).float(), **tol(dtype))
    assert torch.allclose(o.weighted_sum(x, y, 0.8, -1.3).float(), ref_ops.weighted_sum(x, y, 0.8, -1.3).float(), **tol(dtype))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("N,H", [(5, 96), (3, 1000), (40, 2050)])
def test_norm_of_the_pending_term(dtype, N, H):
    o = ops()
    g = torch.Generator().manual_seed(11)
    h = (torch.randn(N, H, generator=g) * 3).cuda()
    delta = (torch.randn(N, H, generator=g) * 5).to(dtype).cuda()
    w, wd = (1 + 0.1 * torch.randn(H, generator=g)).cuda(), (1 + 0.1 * torch.randn(H, generator=g)).cuda()
    h1, h2 = h.clone(), h.clone()
    a = o.add_rmsnorm(h1, delta, w, 1e-6, dtype, wd, 1e-5)
    b = ref_ops.add_rmsnorm(h2, delta, w, 1e-6, dtype, wd, 1e-5)
    assert torch.allclose(h1, h2, atol=1e-5, rtol=1e-5)
    assert torch.allclose(a.float(), b.float(), **tol(dtype))
    rows = torch.tensor([N - 1, 0, N // 2], dtype=torch.int32).cuda()
    assert torch.allclose(o.gather_add(h, delta, rows, wd, 1e-5), ref_ops.gather_add(h, delta, rows, wd, 1e-5), atol=1e-5, rtol=1e-5)
    table = torch.randn(50, H, generator=g).to(dtype).cuda()
    ids = torch.randint(0, 50, (N,), generator=g, dtype=torch.int32).cuda()
    assert torch.allclose(o.embed(ids, table, 7.25), ref_ops.embed(ids, table, 7.25), atol=0, rtol=1e-6)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("H,G,D,Dv", [(4, 2, 16, 16), (3, 1, 32, 48), (2, 2, 40, 24), (6, 2, 64, 64)])
@pytest.mark.parametrize("normed", [True, False])
def test_value_norm_and_padding(dtype, H, G, D, Dv, normed):
    o = ops()
    g = torch.Generator().manual_seed(12)
    qkv = torch.randn(9, H * D + G * D + G * Dv, generator=g).to(dtype).cuda()
    want = ref_ops.value_norm_pad(qkv.clone(), H, G, D, Dv, 1e-5, normed)
    got = o.value_norm_pad(qkv, H, G, D, Dv, 1e-5, normed)
    assert got.shape == want.shape
    assert torch.allclose(got.float(), want.float(), **tol(dtype))


@pytest.mark.parametrize("H,G,D,V", [(4, 2, 64, 128), (2, 2, 16, 24), (3, 1, 40, 33), (6, 2, 32, 40), (10, 5, 64, 256), (1, 1, 1, 1)])
@pytest.mark.parametrize("channel", [False, True])
def test_gated_delta_in_chunks(H, G, D, V, channel):
    """The kernels that run a span in chunks of 64 rows, at every remainder that matters, behind a state and beside spans that
    are walked; decays from next to none to ones that leave nothing of a state within a row, next to each other."""
    o = ops()
    g = torch.Generator().manual_seed(21)
    cols_a = H * D if channel else H
    a_log = torch.log(1 + 15 * torch.rand(H, generator=g)).cuda()
    dt_bias = (torch.randn(cols_a, generator=g) * 2 - 3).cuda()
    norm_w = (1 + 0.1 * torch.randn(V, generator=g)).cuda()
    state_a = (torch.randn(22, H, D, V, generator=g) * 0.3).cuda()
    state_b = state_a.clone()
    for q_lens, impl in (([64, 1, 63, 65], "chunks"), ([129, 300, 2, 128], "chunks"), ([1, 160, 1, 400], None), ([159, 261, 5, 0], None), ([500], None)):
        step = make_step(o, torch.bfloat16, [3] * len(q_lens), q_lens, 8, 256, 5)
        N = sum(q_lens)
        qkv = torch.randn(N, 2 * G * D + H * V, generator=g).bfloat16().cuda()
        a = torch.randn(N, cols_a, generator=g)
        a[N // 3:N // 3 + 20] += 30.0                                  # decays of hundreds of nats a row
        a[N // 2:N // 2 + 40] -= 30.0                                  # and none at all
        a = a.bfloat16().cuda()
        rest = torch.randn(N, H * V + H, generator=g).bfloat16().cuda()
        gate, b = rest[:, :H * V], rest[:, H * V:]
        more = dict(channel_decay=channel, gate_act="sigmoid")
        ya = o.gated_delta(qkv, b, a, gate, a_log, dt_bias, norm_w, 1e-5, state_a, step, H, G, D, V, True, impl=impl, **more)
        yb = ref_ops.gated_delta(qkv, b, a, gate, a_log, dt_bias, norm_w, 1e-5, state_b, step, H, G, D, V, True, **more)
        # the limits of test_gated_delta
        assert torch.allclose(ya.float(), yb.float(), **tol(torch.bfloat16)), (q_lens, float((ya.float() - yb.float()).abs().max()))
        assert torch.allclose(state_a, state_b, atol=1e-4, rtol=1e-4), q_lens
    assert torch.equal(state_a[0], state_b[0])
    keep = state_a.clone()
    o.gated_delta(qkv, b, a, gate, a_log, dt_bias, norm_w, 1e-5, state_a, step, H, G, D, V, False, impl="chunks", **more)
    assert torch.equal(state_a, keep)
    assert o.read_status() == 0


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("V,H,stride,off", [(32, 3, 4, 0), (64, 5, 8, 0), (128, 1, 0, 0), (256, 3, 4, 0), (128, 3, 2, 0), (64, 3, 4, 1), (48, 3, 0, 0)])
def test_gated_rmsnorm_in_fours_and_one_by_one(dtype, V, H, stride, off):
    """Head sizes that are read four columns a load, with rows on and off such a load's boundary, and one that is not; item counts that
    fill no block.  32-bit sums of V terms: 1e-5; bfloat16 results round at 2^-9."""
    from zig_ai_b200.kernels import ops as o
    o.require(extra=("gated_delta",))
    g = torch.Generator().manual_seed(V + H)
    for N, with_w, act in ((1, True, 0), (37, False, 1), (130, True, 0)):
        x = torch.randn(N, H, V, generator=g).cuda()
        w = (1 + 0.1 * torch.randn(V, generator=g)).cuda() if with_w else None
        gs = H * V + stride
        gate = torch.randn(N * gs + off, generator=g).to(dtype).cuda()[off:]
        out = torch.empty(N, H, V, dtype=dtype, device="cuda")
        code = o._fn("gated_delta", "zai_gated_rmsnorm")(out.data_ptr(), x.data_ptr(), o._ptr(w), gate.data_ptr(), gs, o._dt(out), 1e-5, N, H, V, act,
                                                          o._stream())
        assert code == 0
        gv = gate.view(N, gs)[:, :H * V].reshape(N, H, V).double()
        s = torch.sigmoid(gv)
        want = x.double() * torch.rsqrt((x.double() ** 2).mean(-1, keepdim=True) + 1e-5) * (w.double() if with_w else 1) * (s if act else gv * s)
        bound = 1e-5 if dtype is torch.float32 else 2.0 ** -8
        assert ((out.double() - want).abs() <= bound * (want.abs() + 1e-3)).all()
    assert o.read_status() == 0


def delta_inputs(H, G, D, V, N, channel, g):
    cols_a = H * D if channel else H
    a_log, dt_bias = torch.log(1 + 15 * torch.rand(H, generator=g)).cuda(), (torch.randn(cols_a, generator=g) - 3).cuda()
    qkv, a = torch.randn(N, 2 * G * D + H * V, generator=g).bfloat16().cuda(), torch.randn(N, cols_a, generator=g).bfloat16().cuda()
    gate, b = torch.randn(N, H * V, generator=g).bfloat16().cuda(), torch.randn(N, H, generator=g).bfloat16().cuda()
    return qkv, b, a, gate, a_log, dt_bias, torch.ones(V).cuda()


@pytest.mark.parametrize("H,G,D,V", [(16, 8, 64, 128), (16, 4, 40, 72), (16, 16, 64, 256), (16, 8, 64, 64)])
def test_gated_delta_in_few_chunks_and_in_many(H, G, D, V):
    """Few chunks are made by two blocks each (heads of more than 64 values), many by one: a request's rows and state are the same, to the
    bit, and one of 130 rows is the reference's within the limits of test_gated_delta."""
    o = ops()
    g = torch.Generator().manual_seed(29)
    q_lens = [130, 900, 700]
    qkv, b, a, gate, a_log, dt_bias, norm_w = delta_inputs(H, G, D, V, sum(q_lens), False, g)
    state = (torch.randn(6, H, D, V, generator=g) * 0.3).cuda()

    def run(at, lens, n, **kw):
        st = state.clone()
        step = make_step(o, torch.bfloat16, [3] * len(lens), lens, 64, 64, 5)
        y = at.gated_delta(qkv[:n].contiguous(), b[:n].contiguous(), a[:n].contiguous(), gate[:n].contiguous(), a_log, dt_bias, norm_w, 1e-5, st,
                           step, H, G, D, V, True, **kw)
        return y[:130].float(), st[1]
    alone, many, want = run(o, [130], 130, impl="chunks"), run(o, q_lens, sum(q_lens), impl="chunks"), run(ref_ops, [130], 130)
    assert torch.equal(alone[0], many[0]) and torch.equal(alone[1], many[1])
    assert torch.allclose(alone[0], want[0], **tol(torch.bfloat16)) and torch.allclose(alone[1], want[1], atol=1e-4, rtol=1e-4)
    assert o.read_status() == 0


@pytest.mark.parametrize("H,G,D,V", [(4, 2, 64, 128), (2, 2, 24, 40)])
@pytest.mark.parametrize("channel", [False, True])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_gated_delta_in_chunks_and_values_that_are_not_finite(H, G, D, V, channel, bad):
    """A value (or a key) that is not finite reaches its own heads from its own row on, and nothing else."""
    o = ops()
    g = torch.Generator().manual_seed(23)
    step = make_step(o, torch.bfloat16, [3, 3], [200, 70], 8, 256, 5)
    qkv, *rest = delta_inputs(H, G, D, V, 270, channel, g)
    run = lambda rows: o.gated_delta(rows, *rest, 1e-5, torch.zeros(5, H, D, V).cuda(), step, H, G, D, V, True, channel_decay=channel, impl="chunks").view(270, H, V)
    want = run(qkv)
    assert torch.isfinite(want).all()
    for r in (0, 1, 7, 8, 15, 16, 30, 63, 64, 100, 199):
        for col, heads in ((2 * G * D + V // 2, [0]), (G * D, list(range(H // G)))):       # a value of head 0; a key of the first key head
            dirty = qkv.clone()
            dirty[r, col] = bad
            got = run(dirty)
            hit = torch.zeros(270, H, dtype=torch.bool)
            hit[r:200, heads] = True
            assert torch.equal(got[~hit], want[~hit]), (r, col)
            assert not torch.isfinite(got[hit]).all(1).any(), (r, col)
    assert o.read_status() == 0


@pytest.mark.parametrize("channel", [False, True])
def test_gated_delta_in_chunks_with_a_unit_norm_without_epsilon(channel):
    """A span whose last chunk is not full: its spare rows are zeros, which a norm without an epsilon would divide by zero."""
    o = ops()
    g = torch.Generator().manual_seed(24)
    H, G, D, V = 4, 2, 64, 128
    step = make_step(o, torch.bfloat16, [3, 3], [100, 65], 8, 256, 5)
    inputs = delta_inputs(H, G, D, V, 165, channel, g)
    state_a = (torch.randn(5, H, D, V, generator=g) * 0.3).cuda()
    state_b = state_a.clone()
    ya = o.gated_delta(*inputs, 1e-5, state_a, step, H, G, D, V, True, unit_eps=0.0, channel_decay=channel, impl="chunks")
    yb = ref_ops.gated_delta(*inputs, 1e-5, state_b, step, H, G, D, V, True, unit_eps=0.0, channel_decay=channel)
    assert torch.allclose(ya.float(), yb.float(), **tol(torch.bfloat16))
    assert torch.allclose(state_a, state_b, atol=1e-4, rtol=1e-4)


@pytest.mark.parametrize("dtype", DTYPES)
def test_selective_scan_with_rates_that_overflow(dtype):
    """exp(A_log) beyond the largest number: the state is gone after each row (as by any rate that large), and rows that fill up a tile
    change nothing."""
    o = ops()
    g = torch.Generator().manual_seed(25)
    I, S, R = 32, 16, 4
    step = make_step(o, dtype, [3, 3], [5, 66], 8, 256, 5)
    w_dt, b_dt, d = (torch.randn(I, R, generator=g) * 0.5).to(dtype).cuda(), (torch.randn(I, generator=g) * 0.5).cuda(), torch.randn(I, generator=g).cuda()
    x, proj, z = (torch.randn(71, n, generator=g).to(dtype).cuda() for n in (I, R + 2 * S, I))
    out = []
    for rate in (100.0, 30.0):                                 # e^100 is infinite in 32 bits, e^30 is not; both leave nothing
        a_log = (torch.randn(I, S, generator=torch.Generator().manual_seed(1)) * 0.5).cuda()
        a_log[::3] = rate
        state = torch.randn(5, I, S, generator=torch.Generator().manual_seed(2)).cuda()
        out.append((o.selective_scan(x, proj, z, w_dt, b_dt, a_log, d, state, step, R, True), state))
    assert torch.isfinite(out[0][0]).all() and torch.isfinite(out[0][1]).all()
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])


def same_alone_and_beside(run, lens, others):
    """run(q_lens, rows) -> (output rows, states by request) of a step whose requests hold the given rows of the inputs.  A request's rows
    alone, in front of, between and behind others, and in a step that is laid out like a captured one (spans without rows among them)
    must give the same bits."""
    for n in lens:
        want, state = run([n], [0], None)
        for q_lens in others:
            for at in range(len(q_lens) + 1):
                spans = q_lens[:at] + [n] + q_lens[at:]
                first = sum(spans[:at])
                for captured in (None, 1):
                    got, states = run(spans, [200 + i if i != at else 0 for i in range(len(spans))], captured)
                    assert torch.equal(got[first:first + n], want), (n, spans, at, captured)
                    assert torch.equal(states[at], state[0]), (n, spans, at, captured)


@pytest.mark.parametrize("H,G,D,V", [(16, 8, 64, 128), (4, 2, 16, 32), (32, 16, 64, 64)])
@pytest.mark.parametrize("channel", [False, True])
def test_gated_delta_does_not_depend_on_neighbours_or_capture(H, G, D, V, channel):
    o = ops()
    g = torch.Generator().manual_seed(26)
    most = 1100
    qkv, b, a, gate, a_log, dt_bias, norm_w = delta_inputs(H, G, D, V, most, channel, g)
    first = (torch.randn(H, D, V, generator=g) * 0.3).cuda()

    def run(q_lens, shift, captured):
        step = make_step(o, torch.bfloat16, [3] * len(q_lens), q_lens, 8, 2 * sum(q_lens) // 8 + 8 * len(q_lens) + 8, 5)
        if captured:
            step.attn_tiles = sum(q_lens) // 128 + len(q_lens)
        rows = torch.cat([(torch.arange(n) + k) % most for n, k in zip(q_lens, shift)]).cuda()
        state = first.repeat(len(q_lens) + 2, 1, 1, 1)
        y = o.gated_delta(qkv[rows], b[rows], a[rows], gate[rows], a_log, dt_bias, norm_w, 1e-5, state, step, H, G, D, V, True, channel_decay=channel)
        return y, state[1:]
    same_alone_and_beside(run, (2, 5, 64, 127, 128, 130, 256, 700), ([2, 130], [1, 0, 600], [128, 128, 128]))


def test_recurrences_in_chunks_beside_very_many_requests():
    """More requests than a grid's second and third dimension hold."""
    o = ops()
    o.require(extra=("mlstm",))
    g = torch.Generator().manual_seed(27)
    q_lens = [1] * 65600 + [300]
    N = sum(q_lens)
    step = make_step(o, torch.bfloat16, [0] * len(q_lens), q_lens, 8, len(q_lens) + 100, 5)
    y = torch.randn(N, 6 * 8 + 2, generator=g).bfloat16().cuda()
    one = torch.ones(1).cuda()
    outs = []
    for impl in ("walk", None):
        state = torch.zeros(len(q_lens) + 1, 1, 9, 17).cuda()
        outs.append((o.mlstm(y, [0, 8, 16, 32, 48, 49], one, 3 * one, 11.0, torch.ones(16).cuda(), 1e-5, state, step, 1, 8, 16, True, impl=impl), state))
        state = torch.zeros(len(q_lens) + 1, 1, 8, 16).cuda()
        outs.append((o.gated_delta(y[:, :32], y[:, 48:49], y[:, 49:], y[:, 32:48], one, one, torch.ones(16).cuda(), 1e-5, state, step, 1, 1, 8, 16, True, impl=impl), state))
    for (a, sa), (b, sb) in zip(outs[:2], outs[2:]):
        assert torch.equal(a[:65600], b[:65600]) and torch.equal(sa[1:65601], sb[1:65601])
        assert torch.allclose(a.float(), b.float(), **tol(torch.bfloat16)) and torch.allclose(sa, sb, atol=1e-4, rtol=1e-4)
    assert o.read_status() == 0


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("I,S,R", [(96, 16, 8), (36, 12, 4), (68, 4, 4), (20, 28, 8), (24, 64, 8), (20, 100, 8), (12, 200, 4), (256, 16, 16)])
@pytest.mark.parametrize("impl", [None, "chunks"])
def test_selective_scan_of_spans_in_fours(dtype, I, S, R, impl):
    """Rows that are read four values a load (channels, states and strides in fours), at the remainders of tiles of 32 and 64 rows, of
    the channels of a block and of chunks of 512 rows, beside single tokens and a span without rows."""
    o = ops()
    g = torch.Generator().manual_seed(28)
    w_dt, b_dt, d = (torch.randn(I, R, generator=g) * 0.5).to(dtype).cuda(), (torch.randn(I, generator=g) * 0.5 - 1).cuda(), torch.randn(I, generator=g).cuda()
    a_log = (torch.randn(I, S, generator=g) * 0.5 - 1).cuda()
    state_a = torch.randn(9, I, S, generator=g).cuda()
    state_b = state_a.clone()
    for q_lens in ([2, 1, 61, 64, 3], [1, 129, 0, 300], [63, 65, 1, 1], [32, 33], [511, 1, 512], [513, 2, 1025]):
        step = make_step(o, dtype, [3] * len(q_lens), q_lens, 8, 600, 5)
        N = sum(q_lens)
        x, proj, z = (torch.randn(N, n, generator=g).to(dtype).cuda() for n in (I, R + 2 * S, I))
        ya = o.selective_scan(x, proj, z, w_dt, b_dt, a_log, d, state_a, step, R, True, impl=impl)
        yb = ref_ops.selective_scan(x, proj, z, w_dt, b_dt, a_log, d, state_b, step, R, True)
        # the limits of test_selective_scan
        assert torch.allclose(ya.float(), yb.float(), **tol(dtype)), (q_lens, float((ya.float() - yb.float()).abs().max()))
        assert torch.allclose(state_a, state_b, atol=1e-4, rtol=1e-4), (q_lens, float((state_a - state_b).abs().max()))
        state_a.copy_(state_b)
    keep = state_a.clone()
    o.selective_scan(x, proj, z, w_dt, b_dt, a_log, d, state_a, step, R, False, impl=impl)
    assert torch.equal(state_a, keep)
    assert o.read_status() == 0


def test_selective_scan_does_not_depend_on_neighbours_or_capture():
    o = ops()
    g = torch.Generator().manual_seed(29)
    I, S, R, most, dtype = 48, 16, 4, 3000, torch.bfloat16
    w_dt, b_dt, d = (torch.randn(I, R, generator=g) * 0.5).to(dtype).cuda(), (torch.randn(I, generator=g) * 0.5 - 1).cuda(), torch.randn(I, generator=g).cuda()
    a_log, first = (torch.randn(I, S, generator=g) * 0.5 - 1).cuda(), torch.randn(I, S, generator=g).cuda()
    x, proj, z = (torch.randn(most, n, generator=g).to(dtype).cuda() for n in (I, R + 2 * S, I))

    def run(q_lens, shift, captured):
        step = make_step(o, dtype, [3] * len(q_lens), q_lens, 8, 2 * sum(q_lens) // 8 + 8 * len(q_lens) + 8, 5)
        if captured:
            step.attn_tiles = sum(q_lens) // 128 + len(q_lens)
        rows = torch.cat([(torch.arange(n) + k) % most for n, k in zip(q_lens, shift)]).cuda()
        state = first.repeat(len(q_lens) + 2, 1, 1)
        return o.selective_scan(x[rows], proj[rows], z[rows], w_dt, b_dt, a_log, d, state, step, R, True), state[1:]
    same_alone_and_beside(run, (2, 300, 2047, 2048, 2600), ([2, 130], [1, 0, 2100]))
