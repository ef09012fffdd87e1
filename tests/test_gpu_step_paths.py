"""Kernels and dispatch rules of prefill and decode steps at the sizes where they can go wrong, on the GPU."""
import pytest
import torch

from atlas_b200 import quant as Q
from atlas_b200.config import PRESETS, EngineConfig
from atlas_b200.engine import LLMEngine
from atlas_b200.layers.moe import ExpertWeights
from atlas_b200.models import ForwardBatch, build_model
from atlas_b200.ops import reference as ref

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _rel(a, b):
    a, b = a.double(), b.double()
    return float((a - b).norm() / b.norm().clamp_min(1e-30))


@pytest.fixture(scope="module")
def K():
    from atlas_b200.ops import cuda as k
    k.load()
    return k


# ----------------------------------------------------------------------------- experts on live rows
def _fp8(x):
    q, s = Q.per_token_group_quant_fp8(x)
    return (q.float().view(x.shape[0], -1, 128) * s[..., None]).view(x.shape)


def _fp8_experts(x, ex, w, ids, lo):
    """The weighted sum over a token's experts, with activations rounded to FP8 and intermediate rows to bf16."""
    w13, w2 = ex.dequantized()
    y, xq = torch.zeros(x.shape, device=DEV), _fp8(x)
    for e in range(w13.shape[0]):
        t, j = (ids == e + lo).nonzero(as_tuple=True)
        if t.numel():
            g, u = (xq[t] @ w13[e].float().t()).bfloat16().float().chunk(2, -1)
            o = _fp8((torch.nn.functional.silu(g) * u).bfloat16()) @ w2[e].float().t()
            y.index_add_(0, t, o.bfloat16().float() * w[t, j].float()[:, None])
    return y


@pytest.mark.parametrize("T,E,hot", [(1, 512, False), (3, 8, False), (47, 64, False), (130, 4, False), (130, 16, True), (257, 8, True)])
def test_expert_products_touch_live_rows_only(K, T, E, hot):
    """FP8 experts with no, one, a few and more than a tile of rows each, against an oracle that rounds where the kernels do.  What is
    left: rows rounded to bf16 (2^-9), and where another order of the sums turns a group's largest bf16 value, a scale that is
    2^-8 off, which moves up to one in 16 of the group's values to the next FP8 number (a step of 2^-3 to 2^-4): sqrt(1 / 16) * 0.09
    = 0.02 of that row."""
    torch.manual_seed(T + E)
    H, I, k = 256, 128, 3
    ex = ExpertWeights.from_dense((torch.randn(E, 2 * I, H, device=DEV) * 0.05).bfloat16(), (torch.randn(E, H, I, device=DEV) * 0.05).bfloat16(),
                                  "fp8_block")
    logits = torch.randn(T, E, device=DEV)
    if hot:
        logits[:, 1] += 20.0                       # one expert gets every token: full tiles and a remainder
    w, ids = ref.moe_route(logits, k, True)
    x = torch.randn(T, H, device=DEV).bfloat16()
    got = K.moe_forward(x, w.contiguous(), ids.contiguous(), ex, 0, None, "auto")
    assert K.check_status() == 0
    assert _rel(got, _fp8_experts(x, ex, w, ids, 0)) < 0.02
    # a slice of the experts: pairs of the others take no row
    lo, n = E // 4, E // 2
    part = ExpertWeights("fp8_block", ex.w13[lo:lo + n].contiguous(), ex.w2[lo:lo + n].contiguous(), ex.w13_scale[lo:lo + n].contiguous(),
                         ex.w2_scale[lo:lo + n].contiguous())
    got = K.moe_forward(x, w.contiguous(), ids.contiguous(), part, lo, None, "auto")
    want = _fp8_experts(x, part, w, ids, lo)
    assert _rel(got, want) < 0.02 if float(want.abs().max()) > 0 else float(got.abs().max()) == 0


@pytest.mark.parametrize("T,E,H,I", [(30, 4, 256, 128), (60, 4, 256, 128), (300, 3, 4096, 2112)])
def test_bf16_expert_products_by_copy_size_and_order(K, T, E, H, I):
    """Rows copied 32, 64 and 128 at a time (15, 30 and 200 rows an expert), and experts of 34 MB (row tiles first): against an oracle that rounds
    where the kernels do; what is left is the last rounding to bf16 and the few values before it that another order of the sums turns."""
    torch.manual_seed(T + H)
    ex = ExpertWeights.from_dense((torch.randn(E, 2 * I, H, device=DEV) * 0.02).bfloat16(), (torch.randn(E, H, I, device=DEV) * 0.02).bfloat16(), "dense")
    w, ids = ref.moe_route(torch.randn(T, E, device=DEV), 2, True)
    x = torch.randn(T, H, device=DEV).bfloat16()
    got = K.moe_forward(x, w.contiguous(), ids.contiguous(), ex, 0, None, "auto")
    assert K.check_status() == 0
    want = torch.zeros(T, H, device=DEV)
    for e in range(E):
        t, j = (ids == e).nonzero(as_tuple=True)
        g, u = (x[t].double() @ ex.w13[e].double().t()).bfloat16().float().chunk(2, -1)
        o = (torch.nn.functional.silu(g) * u).bfloat16().double() @ ex.w2[e].double().t()
        want.index_add_(0, t, o.bfloat16().float() * w[t, j].float()[:, None])
    assert _rel(got, want) < 2 ** -8


@pytest.mark.parametrize("T,k", [(75, 4), (1023, 4), (1024, 4), (2731, 3)])
def test_expert_row_lists(K, T, k):
    """align: every routed pair has a row of its own inside its expert's segment, and the tiles say how many rows live (one CTA; a
    cluster from 4096 pairs on, with a remainder behind the last four ids)."""
    torch.manual_seed(0)
    E, lo, n = 32, 8, 16
    ids = torch.stack([torch.randperm(E)[:k] for _ in range(T)]).int().to(DEV)
    tiles = T * k // 128 + min(T * k, n)
    slot, rows = torch.empty(T * k, dtype=torch.int32, device=DEV), torch.full((tiles * 128,), -7, dtype=torch.int32, device=DEV)
    te, tr, un, nt = (torch.zeros(m, dtype=torch.int32, device=DEV) for m in (tiles, tiles, tiles, 2))
    K._check(K.lib().atlas_moe_align(ids.data_ptr(), T, k, lo, n, slot.data_ptr(), rows.data_ptr(), te.data_ptr(), tr.data_ptr(), un.data_ptr(), nt.data_ptr(),
                                     tiles * 128, K._status_ptr[K._dev(ids)], K._stream()), "moe_align")
    live, units = nt.tolist()
    assert int(tr[:live].sum()) == int(((ids >= lo) & (ids < lo + n)).sum())
    flat, slot, te, tr, rows = ids.flatten().tolist(), slot.tolist(), te.tolist(), tr.tolist(), rows.tolist()
    used = [s for s in slot if s >= 0]
    assert len(set(used)) == len(used)
    for i, (e, s) in enumerate(zip(flat, slot)):
        assert (s >= 0) == (lo <= e < lo + n)
        if s >= 0:
            assert te[s // 128] == e - lo and s % 128 < tr[s // 128] and rows[s] == i // k
    left, starts = list(range(live)), un[:units].tolist()             # units: pairs of tiles of one expert from its first on
    for t in starts:
        left.remove(t)
        if t + 1 < live and te[t + 1] == te[t]:
            left.remove(t + 1)
    assert not left
    for t in range(live):
        assert all(r == -1 for r in rows[t * 128 + tr[t]:(t + 1) * 128])


@pytest.mark.parametrize("E,k,dtype", [(33, 5, torch.bfloat16), (64, 8, torch.float32), (256, 8, torch.bfloat16), (257, 32, torch.bfloat16),
                                       (512, 10, torch.bfloat16), (513, 10, torch.float32), (1024, 4, torch.bfloat16)])
def test_route_picks_the_largest(K, E, k, dtype):
    """Largest logits first, the lowest expert among equal ones (coarse logits, so that many are), minus infinity last; weights sum to 1."""
    torch.manual_seed(E)
    logits = (torch.randn(19, E, device=DEV) * 4).round().div(2).to(dtype)
    logits[3] = -1.5
    logits[4, k:] = -float("inf")
    w, ids = K.moe_route(logits, k, True, "softmax")
    order = torch.sort(logits.double(), dim=-1, descending=True, stable=True)
    assert torch.equal(ids.long(), order.indices[:, :k])
    want = order.values[:, :k].softmax(-1)
    assert float((w.double() - want).abs().max()) < 1e-5


@pytest.mark.parametrize("T,H,D", [(1, 3, 128), (7, 5, 128), (600, 31, 128), (513, 32, 128), (5, 3, 96), (8193, 32, 128)])
def test_gated_norm_of_heads(K, T, H, D):
    torch.manual_seed(T)
    x, z, w = (torch.randn(*s, device=DEV).bfloat16() for s in ((T, H, D), (T, H, D), (D,)))
    y = K.gated_rmsnorm(x, z, w, 1e-6).double()
    xd = x.double()
    want = xd * torch.rsqrt(xd.square().mean(-1, keepdim=True) + 1e-6) * w.double() * torch.nn.functional.silu(z.double())
    assert float(((y - want).abs() / (want.abs() + 1e-3)).max()) < 2 ** -8


@pytest.mark.parametrize("T,I", [(3, 512), (259, 128), (300, 512), (257, 2304), (1000, 384)])
def test_silu_rows_share_blocks(K, T, I):
    """Rows by index with gaps, several to a block: each is what it is alone, others stay."""
    torch.manual_seed(T)
    gu = torch.randn(T, 2 * I, device=DEV).bfloat16()
    rows = torch.randperm(T)[:T - 1].int().to(DEV)
    rows[::5] = -1
    q, s = torch.zeros(T, I, dtype=torch.uint8, device=DEV), torch.zeros(I // 128, T, device=DEV)
    K._check(K.lib().atlas_silu_mul(gu.data_ptr(), 2 * I, rows.numel(), I, None, 0, q.data_ptr(), I, s.data_ptr(), T, rows.data_ptr(), K._stream()), "silu_mul")
    one, sc = K.silu_mul(gu[:200].contiguous(), quant=True)
    got = torch.zeros(T, dtype=torch.bool, device=DEV)
    got[rows[rows >= 0].long()] = True
    m = min(200, T)
    live = got[:m]
    assert torch.equal(q[:m][live], one[:m].view(torch.uint8)[live]) and torch.equal(s[:, :m].t()[live], sc[:m][live])
    assert int(q[~got].sum()) == 0 and float(s.t()[~got].abs().sum()) == 0


# ----------------------------------------------------------------------------- NVFP4 products of two row tiles a unit
def _row_lists(K, ids, n):
    """Row lists of ``n`` experts: (slot of every pair, tile_expert, unit_tile, num_tiles, rows of the buffer)."""
    T, k = ids.shape
    tiles = T * k // 128 + min(T * k, n)
    slot, rows = torch.empty(T * k, dtype=torch.int32, device=DEV), torch.empty(tiles * 128, dtype=torch.int32, device=DEV)
    te, tr, un, nt = (torch.zeros(m, dtype=torch.int32, device=DEV) for m in (tiles, tiles, tiles, 2))
    K._check(K.lib().atlas_moe_align(ids.data_ptr(), T, k, 0, n, slot.data_ptr(), rows.data_ptr(), te.data_ptr(), tr.data_ptr(), un.data_ptr(), nt.data_ptr(),
                                     tiles * 128, K._status_ptr[K._dev(ids)], K._stream()), "moe_align")
    return slot.long(), te, un, nt, tiles * 128


def _nvfp4(g, E, N, H):
    """Random stack: codes, block scales, a global scale per row."""
    return (torch.randint(0, 256, (E, N, H // 2), generator=g, device=DEV, dtype=torch.uint8),
            (torch.rand(E, N, H // 16, generator=g, device=DEV) + 0.5).to(torch.float8_e4m3fn), torch.rand(E * N, generator=g, device=DEV) * 0.02 + 0.005)


def _nvfp4_value(w, e, rows):
    lut = torch.tensor([0, 0.5, 1, 1.5, 2, 3, 4, 6], dtype=torch.float64, device=DEV)
    lut = torch.cat([lut, -lut])
    v = torch.stack([lut[(w[0][e] & 15).long()], lut[(w[0][e] >> 4).long()]], -1).flatten(1)
    return v * w[1][e].double().repeat_interleave(16, 1) * w[2][e * rows:(e + 1) * rows].double()[:, None]


def _grouped(K, a, w, N, H, te, un, nt, hint, sms):
    c = torch.zeros(a.shape[0], N, dtype=torch.bfloat16, device=DEV)
    E = w[0].shape[0]
    K._check(K.lib().atlas_gemm_w4a16_grouped(a.data_ptr(), w[0].data_ptr(), w[1].data_ptr(), w[2].data_ptr(), c.data_ptr(), a.shape[0], N, H, E, H, N, 128,
                                              te.data_ptr(), un.data_ptr(), nt.data_ptr(), hint, sms, K._status_ptr[K._dev(a)], K._stream()), "w4_grouped")
    return c


@pytest.mark.parametrize("counts", [[1, 128, 129, 256], [257, 0, 640, 300], [513, 127, 1, 0], [385]])
@pytest.mark.parametrize("N,H", [(128, 64), (384, 1088)])
def test_nvfp4_products_of_two_row_tiles(K, counts, N, H):
    """Experts with no, one, two, three and five tiles, last tiles of one row: pairs of tiles (``hint`` above 128) against one tile a unit, the
    same bits on live rows (every accumulator gets the same MMAs in the same order), and against 64 bits (results are rounded to bf16, 2^-9).
    Eight CTAs walk over all units, so rings and accumulators go round many times."""
    from atlas_b200.ops import cuda_ext
    cuda_ext.bind(K.lib())
    g = torch.Generator(device=DEV).manual_seed(sum(counts) + N)
    E = len(counts)
    ids = torch.cat([torch.full((n,), e) for e, n in enumerate(counts)]).int()
    ids = ids[torch.randperm(len(ids))].to(DEV).view(-1, 1)
    slot, te, un, nt, rows = _row_lists(K, ids, E)
    w = _nvfp4(g, E, N, H)
    a = torch.randn(rows, H, generator=g, device=DEV).bfloat16()
    one, two = (_grouped(K, a, w, N, H, te, un, nt, hint, 8) for hint in (0, 129))
    assert K.check_status() == 0
    assert torch.equal(one[slot], two[slot])
    for e, n in enumerate(counts):
        r = slot[ids[:, 0] == e]
        if n:
            assert _rel(two[r], a[r].double() @ _nvfp4_value(w, e, N).t()) < 2 ** -9 + 1e-5


def test_nvfp4_products_of_two_row_tiles_at_full_rate(K):
    """Expert products of a large prompt step (the tensor cores then take all of shared memory's bandwidth): the same bits as one tile a
    unit, in every run."""
    from atlas_b200.ops import cuda_ext
    cuda_ext.bind(K.lib())
    g = torch.Generator(device=DEV).manual_seed(7)
    E, sms = 128, K._num_sms[K._dev(torch.empty(1, device=DEV))]
    ids = torch.rand(4500, E, generator=g, device=DEV).topk(8, -1).indices.int().contiguous()
    slot, te, un, nt, rows = _row_lists(K, ids, E)
    for N, H in ((1536, 2048), (2048, 768)):
        w, a = _nvfp4(g, E, N, H), torch.randn(rows, H, generator=g, device=DEV).bfloat16()
        one = _grouped(K, a, w, N, H, te, un, nt, 0, sms)[slot]
        for _ in range(8):
            assert torch.equal(_grouped(K, a, w, N, H, te, un, nt, 281, sms)[slot], one)
    assert K.check_status() == 0


@pytest.mark.parametrize("M,N,Kd,sms", [(257, 128, 64, 2), (300, 200, 192, 4), (512, 136, 2048, 3), (2500, 4096, 1024, 148), (2304, 4032, 512, 148), (1153, 4096, 4096, 148)])
def test_plain_nvfp4_product_of_two_row_tiles(K, M, N, Kd, sms):
    """Odd and even tile counts, rows past M, columns past N: pairs of row tiles against one (taken when there are fewer units than SMs)."""
    from atlas_b200.ops import cuda_ext
    cuda_ext.bind(K.lib())
    g = torch.Generator(device=DEV).manual_seed(M + N)
    w = _nvfp4(g, 1, N, Kd)
    x = torch.randn(M, Kd, generator=g, device=DEV).bfloat16()
    got = []
    for s in (sms, 1 << 20):
        c = torch.zeros(M + 1, N, dtype=torch.bfloat16, device=DEV)
        K._check(K.lib().atlas_gemm_w4a16(x.data_ptr(), w[0].data_ptr(), w[1].data_ptr(), w[2].data_ptr(), c.data_ptr(), M, N, Kd, Kd, N, 128, s,
                                          K._status_ptr[K._dev(x)], K._stream()), "w4")
        got.append(c)
    assert K.check_status() == 0
    assert torch.equal(got[0], got[1]) and float(got[0][M].abs().max()) == 0
    assert _rel(got[0][:M], x.double() @ _nvfp4_value(w, 0, N).t()) < 2 ** -9 + 1e-5


@pytest.mark.parametrize("counts", [[1, 0, 8], [9, 7, 33, 2], [70, 3]])
@pytest.mark.parametrize("H,I", [(256, 256), (4096, 256), (4352, 512)])
def test_small_nvfp4_experts_with_and_without_whole_rows_staged(K, counts, H, I):
    """Tiles around eight rows and more than one pass of 32, K at and behind the longest that is staged whole: both kernels give the same
    bits (the same MMAs in the same order), and 64 bits up to the rounding of intermediate rows and results to bf16 (2^-9 each, the
    first through a product)."""
    from atlas_b200.ops import cuda_ext
    lib = K.lib()
    cuda_ext.bind(lib)
    cuda_ext._bind_small(lib)
    g = torch.Generator(device=DEV).manual_seed(sum(counts) + H)
    E, T = len(counts), sum(counts)
    ids = torch.cat([torch.full((n,), e) for e, n in enumerate(counts)]).int().to(DEV).view(-1, 1)
    tiles = T // 128 + min(T, E)
    slot, rows = torch.empty(T, dtype=torch.int32, device=DEV), torch.empty(tiles * 128, dtype=torch.int32, device=DEV)
    te, tr, nt = (torch.zeros(m, dtype=torch.int32, device=DEV) for m in (tiles, tiles, 2))
    K._check(lib.atlas_moe_align(ids.data_ptr(), T, 1, 0, E, slot.data_ptr(), rows.data_ptr(), te.data_ptr(), tr.data_ptr(), None, nt.data_ptr(), tiles * 128,
                                 K._status_ptr[K._dev(ids)], K._stream()), "moe_align")
    w13, w2 = _nvfp4(g, E, 2 * I, H), _nvfp4(g, E, H, I)
    x = (torch.randn(T, H, generator=g, device=DEV) * 0.1).bfloat16()
    got = []
    for few in (0, 1):
        act, y = (torch.zeros(tiles * 128, n, dtype=torch.bfloat16, device=DEV) for n in (I, H))
        K._check(lib.atlas_moe_small_w4(1, x.data_ptr(), H, rows.data_ptr(), te.data_ptr(), nt.data_ptr(), tiles, w13[0].data_ptr(), w13[1].data_ptr(),
                                        w13[2].data_ptr(), act.data_ptr(), I, H, 2 * I, few, K._stream()), "up")
        K._check(lib.atlas_moe_small_w4(0, act.data_ptr(), I, rows.data_ptr(), te.data_ptr(), nt.data_ptr(), tiles, w2[0].data_ptr(), w2[1].data_ptr(),
                                        w2[2].data_ptr(), y.data_ptr(), H, I, H, few, K._stream()), "down")
        got.append((act[slot.long()], y[slot.long()]))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    for e in range(E):
        r = (ids[:, 0] == e)
        if int(r.sum()):
            gate, up = (x[r].double() @ _nvfp4_value(w13, e, 2 * I).t()).bfloat16().double().chunk(2, -1)
            want = (torch.nn.functional.silu(gate) * up).bfloat16().double() @ _nvfp4_value(w2, e, H).t()
            assert _rel(got[1][1][r], want) < 2 ** -8


@pytest.mark.parametrize("C,ld,off", [(8, 8, 0), (12, 12, 0), (2052, 4104, 4), (1024, 1028, 4), (40, 44, 0), (1023, 1023, 0)])
@pytest.mark.parametrize("taps,rows,silu", [(4, 261, 1), (2, 300, 2), (3, 1031, 1), (1, 257, 0), (4, 6200, 1)])
def test_convolution_of_rows_at_any_alignment(K, C, ld, off, taps, rows, silu):
    """bf16 rows that start on 16, 8 or 2 bytes, two sequences, more and fewer rows than the widest loads are taken for: against 64 bits
    (fp32 sums, a result rounded to bf16)."""
    from atlas_b200.ops import cuda_gdn, cuda_recurrent
    g = torch.Generator(device=DEV).manual_seed(C + rows)
    x = torch.randn(rows, ld + off, generator=g, device=DEV).bfloat16()[:, off:off + C]
    w = (torch.randn(C, taps, generator=g, device=DEV) * 0.5).bfloat16()
    bias = torch.randn(C, generator=g, device=DEV).bfloat16()
    state = torch.randn(2, C, max(1, taps - 1), generator=g, device=DEV).bfloat16()[:, :, :taps - 1].contiguous()
    lens = [rows - 5, 5]
    meta = cuda_gdn._Meta(lens, [1, 0], [True, False], DEV)
    y = torch.zeros(rows, C, dtype=torch.bfloat16, device=DEV)
    cuda_recurrent.conv_silu(x, w, bias, state, meta, y, False, silu=silu)
    for (lo, hi), win in (((0, rows - 5), state[1]), ((rows - 5, rows), torch.zeros_like(state[0]))):
        full = torch.cat([win.double().t(), x[lo:hi].double()])
        want = (full.unfold(0, taps, 1) * w.double()).sum(-1) + bias.double()
        want = torch.nn.functional.silu(want) if silu else want
        assert float(((y[lo:hi].double() - want).abs() / (want.abs() + 1e-2)).max()) < 2 ** -8


# ----------------------------------------------------------------------------- decode graphs of Gated DeltaNet models
@pytest.mark.parametrize("n", [1, 3, 9])
def test_delta_net_decode_graph_equals_eager_steps(K, n):
    """Three decode steps from the same states, replayed and eager (padding rows included): the same bits."""
    cfg = PRESETS["tiny-hybrid"]("bfloat16")
    model = build_model(cfg, device=DEV, with_mtp=False).init_random(0, max_pos=256)
    outs = []
    for graphs in (True, False):
        eng = LLMEngine(model, EngineConfig(max_seq_len=256, num_kv_blocks=64, max_num_seqs=n, max_batch_size=n, use_cuda_graphs=graphs,
                                            enable_prefix_caching=False))
        gen = torch.Generator(device=DEV).manual_seed(5)
        for i, st in eng.cache.states.items():
            st["h"][:n] = torch.randn(st["h"][:n].shape, generator=gen, device=DEV) * 0.1
            st["conv"][:n] = torch.randn(st["conv"][:n].shape, generator=gen, device=DEV).bfloat16()
        for k, v in eng.cache.kv.values():
            k.copy_(torch.zeros(k.shape, device=DEV).to(k.dtype))
            v.copy_(torch.zeros(v.shape, device=DEV).to(v.dtype))
        got = []
        for s in range(3):
            b = ForwardBatch.build([[7 * i + s + 1] for i in range(n)], [4 + s] * n, [[2 * i, 2 * i + 1] for i in range(n)], 16, device=DEV,
                                   state_slots=list(range(n)), has_state=[True] * n)
            with torch.inference_mode():
                got.append(eng.runner.forward(b).clone())
        assert (eng.runner.graph_replays == 3) == graphs
        outs.append(got + [st["h"][:n].clone() for st in eng.cache.states.values()] + [st["conv"][:n].clone() for st in eng.cache.states.values()])
    assert all(torch.equal(a, b) for a, b in zip(*outs))


@pytest.mark.parametrize("short", [False, True])
def test_capture_gives_memory_back_only_where_it_is_short(K, short, monkeypatch):
    """The first step of a batch size pays for two eager passes and a capture, not for a collection and the allocator's cache."""
    import gc
    from atlas_b200 import runner
    calls = []
    total = torch.cuda.mem_get_info()[1]
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda *a: (total // 32 if short else total // 2, total))
    monkeypatch.setattr(gc, "collect", lambda *a: calls.append("collect"))
    monkeypatch.setattr(torch.cuda, "empty_cache", lambda: calls.append("empty"))
    x = torch.arange(8.0, device=DEV)
    graph, y = runner._capture(torch.cuda.Stream(), lambda: x * 2)
    assert gc.isenabled() and calls == (["collect", "empty"] if short else [])
    x.add_(1)
    graph.replay()
    assert torch.equal(y, (torch.arange(8.0, device=DEV) + 1) * 2)
    with pytest.raises(ZeroDivisionError):
        runner._capture(torch.cuda.Stream(), lambda: x * (1 // 0))
    assert gc.isenabled() and float((x + 1).sum()) == 44.0          # the stream is usable again


# ----------------------------------------------------------------------------- chunked delta rule
def _delta_rule(y, a, b, a_log, dt_bias, h, hk, hv, stops):
    """The recurrence in 64 bits: outputs, and the state after every row count in ``stops``."""
    y, a, b, h = y.double(), a.double(), b.double(), h.double().clone()
    n, d, out, kept = y.shape[0], 128, [], {}
    unit = lambda t: t * torch.rsqrt(t.square().sum(-1, keepdim=True) + 1e-6)
    q, k = unit(y[:, :hk * d].view(n, hk, d)) / d ** 0.5, unit(y[:, hk * d:2 * hk * d].view(n, hk, d))
    q, k, v = q.repeat_interleave(hv // hk, 1), k.repeat_interleave(hv // hk, 1), y[:, 2 * hk * d:].view(n, hv, d)
    decay = torch.exp(-torch.exp(a_log.double()) * torch.nn.functional.softplus(a + dt_bias.double()))
    beta = torch.sigmoid(b)
    for t in range(n):
        h = h * decay[t][:, None, None]
        h = h + k[t][:, :, None] * ((v[t] - torch.einsum("hkv,hk->hv", h, k[t])) * beta[t][:, None])[:, None]
        out.append(torch.einsum("hkv,hk->hv", h, q[t]).flatten())
        if t + 1 in stops:
            kept[t + 1] = h.clone()
    return torch.stack(out), kept


@pytest.mark.parametrize("lens,snaps,like", [([1], {}, 0.0), ([64, 63, 65], {}, 0.0), ([300, 1, 128], {0: [(1, 6), (64, 7), (200, 8)], 2: [(128, 9)]}, 0.0),
                                             ([515], {0: [(130, 3)]}, 0.95)])
def test_chunked_delta_rule_against_64_bits(K, lens, snaps, like):
    """Edges of the 64-row chunks, snapshot rows inside and on them, and keys that are nearly the same (``like``: the inverse inside a
    chunk is then far from the identity).  Every product rounds its operands to TF32 (2^-12 in the norm), of which a state and an
    output take about ten in a chain: 2.5e-3; outputs are rounded to bf16 besides (2^-9 at most)."""
    import ctypes
    from atlas_b200.ops import cuda_gdn
    torch.manual_seed(sum(lens))
    hk, hv, d, T, B = 2, 4, 128, sum(lens), len(lens)
    y = torch.randn(T, (2 * hk + hv) * d, device=DEV)
    base = torch.randn(1, hk * d, device=DEV)
    y[:, hk * d:2 * hk * d] = like * base + (1 - like * like) ** 0.5 * y[:, hk * d:2 * hk * d]
    y = y.bfloat16()
    a, b = torch.randn(T, hv, device=DEV).bfloat16(), torch.randn(T, hv, device=DEV).bfloat16()
    a_log, dt_bias = torch.linspace(-3, 2, hv, device=DEV), torch.linspace(-4, 1, hv, device=DEV)
    h0 = torch.randn(12, hv, d, d, device=DEV) * 0.1
    has = [i % 2 == 0 for i in range(B)]
    meta = cuda_gdn._Meta(lens, list(range(B)), has, DEV, snaps)
    h, out, lib = h0.clone(), torch.empty(T, hv * d, dtype=torch.bfloat16, device=DEV), cuda_gdn._lib()
    heads = ctypes.c_int()
    work = torch.empty(lib.atlas_gdn_chunked_bytes(T, B, meta.snaps, hk, hv, ctypes.byref(heads)), dtype=torch.uint8, device=DEV)
    assert heads.value == hv
    K._check(lib.atlas_gdn_chunked(y.data_ptr(), y.stride(0), a.data_ptr(), hv, b.data_ptr(), hv, a_log.data_ptr(), dt_bias.data_ptr(), h.data_ptr(),
                                   out.data_ptr(), hv * d, meta.qsl.data_ptr(), meta.slots.data_ptr(), meta.has.data_ptr(), meta.snap_rows.data_ptr(),
                                   meta.snap_slots.data_ptr(), meta.snaps, T, B, hk, hv, d, d, 1, 1, work.data_ptr(), K._stream()), "gdn_chunked")
    t = 0
    for i, n in enumerate(lens):
        rows = slice(t, t + n)
        t += n
        stops = {r: s for r, s in snaps.get(i, [])}
        want, kept = _delta_rule(y[rows], a[rows], b[rows], a_log, dt_bias, h0[i] * has[i], hk, hv, set(stops) | {n})
        assert _rel(out[rows], want) < 2.5e-3 + 2 ** -9
        assert _rel(h[i], kept[n]) < 2.5e-3
        for r, s in stops.items():
            assert _rel(h[s], kept[r]) < 2.5e-3


def test_chunked_delta_rule_workspace_is_bounded(K):
    """Long steps go through the heads in groups, with the results of one group."""
    import ctypes
    from atlas_b200.ops import cuda_gdn
    lib, heads = cuda_gdn._lib(), ctypes.c_int()
    small = lib.atlas_gdn_chunked_bytes(8192, 1, 0, 16, 32, ctypes.byref(heads))
    assert heads.value == 32 and small <= 256 << 20
    assert lib.atlas_gdn_chunked_bytes(40000, 3, 2, 16, 32, ctypes.byref(heads)) <= 256 << 20 and heads.value == 8
    torch.manual_seed(1)
    hk, hv, d, T = 3, 3, 128, 150000
    assert lib.atlas_gdn_chunked_bytes(T, 1, 0, hk, hv, ctypes.byref(heads)) <= 256 << 20 and heads.value == 1
    y = torch.randn(T, (2 * hk + hv) * d, device=DEV).bfloat16()
    a, b = torch.randn(T, hv, device=DEV).bfloat16(), torch.randn(T, hv, device=DEV).bfloat16()
    a_log, dt_bias = torch.zeros(hv, device=DEV), torch.zeros(hv, device=DEV)
    res = []
    for only in (None, 2):                    # all heads; the last one alone, as a model of one head
        n = hv if only is None else 1
        yy = y if only is None else torch.cat([y[:, (only + i) * d:(only + i + 1) * d] for i in (0, hk, 2 * hk)], 1).contiguous()
        aa, bb = (a, b) if only is None else (a[:, only:only + 1].contiguous(), b[:, only:only + 1].contiguous())
        meta = cuda_gdn._Meta([T], [0], [False], DEV)
        h, out = torch.zeros(1, n, d, d, device=DEV), torch.empty(T, n * d, dtype=torch.bfloat16, device=DEV)
        work = torch.empty(lib.atlas_gdn_chunked_bytes(T, 1, 0, n, n, ctypes.byref(heads)), dtype=torch.uint8, device=DEV)
        K._check(lib.atlas_gdn_chunked(yy.data_ptr(), yy.stride(0), aa.data_ptr(), n, bb.data_ptr(), n, a_log.data_ptr(), dt_bias.data_ptr(),
                                       h.data_ptr(), out.data_ptr(), n * d, meta.qsl.data_ptr(), meta.slots.data_ptr(), meta.has.data_ptr(),
                                       meta.snap_rows.data_ptr(), meta.snap_slots.data_ptr(), 0, T, 1, n, n, d, d, 1, 1, work.data_ptr(), K._stream()), "gdn_chunked")
        res.append((out.view(T, n, d)[:, -1].clone(), h[0, -1].clone()))
    assert torch.equal(res[0][0], res[1][0]) and torch.equal(res[0][1], res[1][1])


@pytest.mark.parametrize("groups", [(2, 1), (1, 1, 1)])
def test_chunked_delta_rule_goes_through_groups_of_heads(K, groups, monkeypatch):
    """Three key heads of two value heads each, two and one or one at a time (a small limit in place of 256 MB): outputs, states and
    snapshots are those of all heads at once, bit for bit, and the recurrence's."""
    import ctypes
    import types
    from atlas_b200.ops import cuda_gdn
    torch.manual_seed(3)
    hk, hv, d, lens, plan = 3, 6, 128, [100, 7, 65], {0: [(30, 4), (64, 5)], 2: [(65, 6)]}
    T, B, lib = sum(lens), len(lens), cuda_gdn._lib()
    C = (2 * hk + hv) * d
    layer = types.SimpleNamespace(hk=hk, hv=hv, dk=d, dv=d, W=4, conv_w=(torch.randn(C, 4, device=DEV) * 0.3).bfloat16(),
                                  A_log=torch.linspace(-2, 2, hv, device=DEV), dt_bias=torch.linspace(-4, 0, hv, device=DEV))
    mixed, a, b = (torch.randn(T, n, device=DEV).bfloat16() for n in (C, hv, hv))
    state = dict(conv=torch.randn(8, C, 3, device=DEV).bfloat16(), h=torch.randn(8, hv, d, d, device=DEV) * 0.1)
    meta = cuda_gdn._Meta(lens, [2, 0, 1], [True, True, False], DEV, plan)
    heads = ctypes.c_int()
    most = cuda_gdn.WORK_LIMIT
    whole = lib.atlas_gdn_chunked_bytes(T, B, meta.snaps, hk, hv, ctypes.byref(heads))
    assert heads.value == hv and whole == lib.atlas_gdn_chunked_bytes_within(most, T, B, meta.snaps, hk, hv, ctypes.byref(heads))
    limit = whole * groups[0] // hk
    assert lib.atlas_gdn_chunked_bytes_within(limit, T, B, meta.snaps, hk, hv, ctypes.byref(heads)) == limit and heads.value == 2 * groups[0]
    assert lib.atlas_gdn_chunked_bytes_within(1, T, B, meta.snaps, hk, hv, ctypes.byref(heads)) == whole // hk and heads.value == 2      # never less
    got = []
    for lim, chunked in ((most, True), (limit, True), (most, False)):
        monkeypatch.setattr(cuda_gdn, "WORK_LIMIT", lim)
        monkeypatch.setattr(cuda_gdn, "USE_CHUNKED", chunked)
        st = {k: v.clone() for k, v in state.items()}
        got.append((cuda_gdn._run(layer, mixed, a, b, meta, st, True), st["h"], st["conv"]))
    assert all(torch.equal(x, y) for x, y in zip(got[0], got[1]))
    assert _rel(got[1][0], got[2][0]) < 1e-2
    for slot in range(8):
        assert _rel(got[1][1][slot], got[2][1][slot]) < 3e-3, slot


# ----------------------------------------------------------------------------- chunk attention of 256-wide heads
@pytest.mark.parametrize("kv", [torch.float8_e4m3fn, torch.bfloat16])
@pytest.mark.parametrize("Hq,Hkv,qlens,ctxs", [(16, 2, [300, 1, 37, 63], [0, 90, 1000, 77]), (8, 2, [64, 65, 129], [64, 63, 0]), (4, 4, [130, 16], [1, 500]),
                                               (16, 1, [40], [200])])
def test_chunk_attention_of_wide_heads(K, kv, Hq, Hkv, qlens, ctxs, monkeypatch):
    """Head dim 256 on the tcgen05 path (64-token KV tiles): edges of query and KV tiles, contexts, several group sizes (16 heads a group is
    taken with a bf16 cache only), beside the general kernel; the bounds are those of the 128-wide heads."""
    from test_gpu_kernels import _attention_case
    args = dict(qlens=qlens, ctxs=ctxs, kv_dtype=kv)
    out, want = _attention_case(K, 256, Hq, Hkv, **args)
    assert K.check_status() == 0
    assert _rel(out, want) < 2e-2
    torch.testing.assert_close(out.float(), want.float(), atol=3e-2, rtol=5e-2)
    monkeypatch.setattr(K, "_TC_PREFILL", False)
    old, _ = _attention_case(K, 256, Hq, Hkv, **args)
    assert _rel(out, want) <= 1.05 * _rel(old, want)
    assert _rel(out, old) < 2e-2


@pytest.mark.parametrize("opts", [dict(window=40), dict(window=64, sinks=True), dict(chunk=96), dict(chunk=64, sinks=True), dict(softcap=5.0, sinks=True),
                                  dict(distance=17), dict(distance=700), dict(distance=9, sinks=True, window=50), dict(distance=30, softcap=8.0)])
@pytest.mark.parametrize("Hq,Hkv", [(4, 4), (6, 2), (16, 2), (20, 1)])
def test_chunk_attention_of_wide_heads_with_every_option(K, Hq, Hkv, opts, monkeypatch):
    """Head dim 256, bf16 cache: windows, chunked visibility, sinks, bounded scores and distance biases (in shared memory and too many for
    it) on the tcgen05 tiles and on the general kernel.  Both round P and the result to bf16, at other places: 2^-8 each at most."""
    g = torch.Generator(device=DEV).manual_seed(Hq)
    qlens, ctxs, D = [130, 5, 64, 33], [0, 300, 63, 127], 256
    nblk = [(c + n + 15) // 16 for c, n in zip(ctxs, qlens)]
    perm, tables, off = torch.randperm(sum(nblk) + 2, generator=g, device=DEV).tolist(), [], 0
    for n in nblk:
        tables.append(perm[off:off + n])
        off += n
    kc, vc = K.alloc_kv_cache(sum(nblk) + 2, 16, Hkv, D, torch.bfloat16, DEV)
    kc.copy_(torch.randn(kc.shape, generator=g, device=DEV).bfloat16())
    vc.copy_(torch.randn(vc.shape, generator=g, device=DEV).bfloat16())
    q = torch.randn(sum(qlens), Hq, D, generator=g, device=DEV).bfloat16()
    sinks = torch.randn(Hq, generator=g, device=DEV) if opts.get("sinks") else None
    reach = opts.get("distance")
    distance = torch.randn(Hq, reach + 1, generator=g, device=DEV) if reach else None
    outs = []
    for tc in (True, False):
        monkeypatch.setattr(K, "_TC_PREFILL", tc)
        fb = ForwardBatch.build([[0] * n for n in qlens], ctxs, tables, 16, device=DEV)
        outs.append(K.paged_attention(q, kc, vc, fb, D ** -0.5, 1.0, 1.0, opts.get("window"), opts.get("chunk", 0), sinks, opts.get("softcap", 0.0), distance))
    assert K.check_status() == 0
    assert _rel(outs[0], outs[1]) < 2 ** -7
    torch.testing.assert_close(outs[0].float(), outs[1].float(), atol=3e-2, rtol=3e-2)


# ----------------------------------------------------------------------------- wide tiles whose last one is cut off
@pytest.mark.parametrize("N", [1990, 2040, 1947])
@pytest.mark.parametrize("form", ["plain", "bias", "unit", "unit_tail", "relu2", "tail", "tail_bias"])
def test_bf16_products_on_cut_off_wide_tiles(K, N, form):
    """38 row tiles of 128 on 256-wide column tiles of which the last one is not whole, through every epilogue, against fp32 products of the
    same bf16 values (fp32 sums; results rounded to bf16: 2^-9, a gated unit's two factors before that)."""
    g = torch.Generator(device=DEV).manual_seed(N)
    M, Kd = 4737, 136
    if form.startswith("unit"):
        N = N // 16 * 16
    assert K.gemm_plan(M, N, Kd, 0, 148)[0] == 256 and N % 256
    x = torch.randn(M, Kd, generator=g, device=DEV).bfloat16()
    w = (torch.randn(N, Kd, generator=g, device=DEV) * 0.1).bfloat16()
    bias = torch.randn(N, generator=g, device=DEV)
    want = x.double() @ w.double().t()
    unit, n_main = (7.0, 1.702, 1.0), N - 80

    def gated(v):
        gate, up = v[:, 0::2].clamp(max=unit[0]), v[:, 1::2].clamp(-unit[0], unit[0])
        return gate * torch.sigmoid(unit[1] * gate) * (up + unit[2])

    if form == "plain":
        pairs = [(K.gemm_bf16(x, w), want)]
    elif form == "bias":
        pairs = [(K.gemm_bf16(x, w, bias=bias), want + bias.double())]
    elif form == "unit":
        pairs = [(K.gemm_bf16(x, w, unit=unit), gated(want))]
    elif form == "unit_tail":
        main, tail = K.gemm_bf16(x, w, unit=unit, n_main=n_main)
        pairs = [(main, gated(want[:, :n_main])), (tail, want[:, n_main:])]
    elif form == "relu2":
        pairs = [(K.gemm_bf16(x, w, relu2_cols=N - 70), torch.cat([want[:, :N - 70].relu().square(), want[:, N - 70:]], 1))]
    else:
        b = bias if form == "tail_bias" else None
        main, tail = K.linear_tail(x, w, N - 77, b)
        full = want + (bias.double() if b is not None else 0.0)
        pairs = [(main, full[:, :N - 77]), (tail, full[:, N - 77:])]
    assert K.check_status() == 0
    for got, ref64 in pairs:
        assert got.shape == ref64.shape and _rel(got, ref64) < (2 ** -9 if got.dtype == torch.bfloat16 else 1e-5)
        assert float((got.double() - ref64)[:, -16:].abs().max()) < 2 ** -6 * float(ref64.abs().max())


@pytest.mark.parametrize("M,N,Kd", [(4737, 1984, 2048), (4737, 2000, 4096), (300, 18432 + 136, 6144)])
def test_fp8_products_on_cut_off_wide_tiles(K, M, N, Kd):
    """Block scales of the last, half or fully missing 128 columns of a wide tile: against 64 bits with the same scales."""
    g = torch.Generator(device=DEV).manual_seed(N)
    xq, xs = K.quant_fp8(torch.randn(M, Kd, generator=g, device=DEV).bfloat16())
    w = torch.randn(N, Kd, generator=g, device=DEV).to(torch.float8_e4m3fn)
    ws = torch.rand((N + 127) // 128, Kd // 128, generator=g, device=DEV) + 0.5
    got = {}
    for bn in (256, 128):
        plan = K.gemm_plan
        try:
            K.gemm_plan = lambda *a: (bn, 1)
            got[bn] = K.gemm_fp8_block(xq, xs, w, ws)
        finally:
            K.gemm_plan = plan
    assert K.check_status() == 0
    assert torch.equal(got[256], got[128])
    rows = torch.tensor([0, 1, M // 2, M - 1], device=DEV)
    a = xq[rows].double().view(4, -1, 128) * xs[rows].double()[..., None]
    b = w.double().view(N, -1, 128) * ws.double().repeat_interleave(128, 0)[:N, :, None]
    assert _rel(got[256][rows], a.flatten(1) @ b.flatten(1).t()) < 2 ** -9
