"""Tensor-core forms of the token-id models' kernels at the sizes where they can go wrong (tile edges, remainders, the
smallest and largest of their ranges), against float64 on the device.  Products of bf16 numbers are exact, their sums are
fp32: the tensor core truncates after every step of 16 products, at most 2^-23 of the running sum each time, and the
truncations of a sum all go one way, half that much on average."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF, F32 = torch.bfloat16, torch.float32


@pytest.fixture(scope="module")
def ops():
    from vila_b200 import ops
    return ops


def rel(a, b):
    return float((a.double() - b).norm() / b.norm().clamp_min(1e-30))


def acc(K):
    """relative error of fp32 sums over K products that are truncated every 16, and of an epilogue's few roundings"""
    return K / 16 * 2.0 ** -24 + 1e-6


def gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def randn(g, *shape, dtype=BF):
    return torch.randn(*shape, generator=g, device="cuda").to(dtype)


@pytest.mark.parametrize("M,N,K", [(1, 128, 8), (8, 1000, 512), (15, 129, 72), (16, 256, 64), (17, 384, 136), (64, 130, 2048),
                                   (65, 257, 448), (128, 128, 200), (129, 640, 1000), (257, 130, 64),
                                   (300, 1408, 2048)])
def test_glinear_plain(ops, M, N, K):
    g = gen(M * 7 + N)
    a, w, b = randn(g, M, K + 8)[:, :K], randn(g, N, K), randn(g, N)
    ref = a.double() @ w.double().T
    assert rel(ops.glinear(a, w, out_dtype=F32), ref) < acc(K)
    assert rel(ops.glinear(a, w, bias=b, act=ops.ACT_RELU2, out_dtype=F32), torch.relu(ref + b.double()) ** 2) < 2 * acc(K)
    assert rel(ops.glinear(a, w), ref) < 2.0 ** -8
    if N % 2 == 0:
        z = ref / K ** 0.5
        want = torch.nn.functional.silu(z[:, 0::2]) * z[:, 1::2]
        assert rel(ops.glinear((a.float() / K ** 0.5).to(BF), w, swiglu=True, out_dtype=F32), want) < 2.0 ** -7   # a is rounded once more
    torch.cuda.synchronize()
    ops.check_waits()


@pytest.mark.parametrize("T,E,top,W,ff", [(3, 8, 2, 128, 128), (8, 32, 4, 256, 192), (40, 5, 3, 136, 200), (200, 33, 2, 256, 264), (520, 4, 2, 320, 136)])
@pytest.mark.parametrize("skew", [False, True])
def test_glinear_routed(ops, T, E, top, W, ff, skew):
    """experts with no rows, with one and with more than a tile; scattered output rows, routing weights, input scales"""
    g = gen(T + E)
    x, up, down = randn(g, T, W), randn(g, E, 2 * ff, W), randn(g, E, W, ff)
    score = torch.rand(T, E, generator=g, device="cuda")
    if skew:
        score[:, 1] += 1.0
        score[:, E - 1] -= 2.0
    idx = score.topk(top, 1).indices.to(torch.int32)
    wt = torch.rand(T, top, generator=g, device="cuda")
    seg, srt = ops.moe_group(idx, E)
    act = ops.glinear(x, up, groups=E, seg=seg, a_rows=srt, a_row_div=top, glu_clamp=(1.702, 7.0), out_dtype=F32)
    part = ops.glinear(act.to(BF), down, groups=E, seg=seg, o_rows=srt, row_scale=wt.view(-1), out_dtype=F32, out_rows_total=T * top)
    scaled = ops.glinear(x, up, groups=E, seg=seg, a_rows=srt, a_row_div=top, in_scale=wt.view(-1), out_dtype=F32)
    e, pair = idx.view(-1)[srt.long()].long(), srt.long()
    z = torch.einsum("rk,rnk->rn", x.double()[pair // top], up.double()[e])
    gt, u = z[:, 0::2].clamp_max(7.0), z[:, 1::2].clamp(-7.0, 7.0)
    assert rel(act, gt * torch.sigmoid(1.702 * gt) * (u + 1)) < 2 * acc(W)
    assert rel(scaled, z * wt.view(-1)[pair].double()[:, None]) < acc(W)
    want = torch.empty(T * top, W, device="cuda", dtype=torch.float64)
    want[pair] = torch.einsum("rk,rnk->rn", act.to(BF).double(), down.double()[e]) * wt.view(-1)[pair].double()[:, None]
    assert rel(part, want) < acc(ff)


@pytest.mark.parametrize("M", [1, 20, 150])
def test_glinear_batched(ops, M):
    """per-head projections: column groups of A and of the output"""
    g, H, K, N = gen(M), 6, 136, 128
    a, w = randn(g, M, H * K), randn(g, H, N, K)
    ref = torch.einsum("mhk,hnk->mhn", a.double().view(M, H, K), w.double()).reshape(M, H * N)
    assert rel(ops.glinear(a, w, groups=H, a_group_off=K, o_group_off=N, out_dtype=F32), ref) < acc(K)


@pytest.mark.parametrize("K", [256, 2048, 8192])
@pytest.mark.parametrize("positive", [False, True])
def test_glinear_few_rows_sum_in_fp32(ops, K, positive):
    """up to 16 rows, or 64 routed pairs: a lane's chain of K / 32 rounded multiply-adds (errors both ways) and five steps of
    a tree, whatever the number of rows and outputs is"""
    g = gen(K)
    tol = (K / 32) ** 0.5 * 2.0 ** -25 + 5 * 2.0 ** -25
    data = (lambda *s: randn(g, *s).abs()) if positive else (lambda *s: randn(g, *s))
    for N in (130, 6002, 12004):
        a, w = data(16, K), data(N, K)
        ref, alone = a.double() @ w.double().T, ops.glinear(a[:1], w, out_dtype=F32)
        for M in (1, 2, 3, 5, 8, 9, 16):
            got = ops.glinear(a[:M], w, out_dtype=F32)
            assert rel(got, ref[:M]) < tol and torch.equal(got[:1], alone)
            z = torch.nn.functional.silu(ref[:M, 0::2]) * ref[:M, 1::2]
            assert rel(ops.glinear(a[:M], w, swiglu=True, out_dtype=F32), z) < 3 * tol + 1e-6
    for T, E, top in ((3, 8, 2), (16, 32, 4), (64, 4, 1), (32, 2, 2), (20, 1, 1)):
        x, w = data(T, K), data(E, 256, K)
        idx = torch.rand(T, E, generator=g, device="cuda").topk(top, 1).indices.to(torch.int32)
        seg, srt = ops.moe_group(idx, E)
        got = ops.glinear(x, w, groups=E, seg=seg, a_rows=srt, a_row_div=top, out_dtype=F32)
        e, tok = idx.view(-1)[srt.long()].long(), srt.long() // top
        assert rel(got, torch.einsum("rk,rnk->rn", x.double()[tok], w.double()[e])) < tol


def test_glinear_one_row_at_every_tile_size(ops):
    """the kernels of few, some and many rows cut K differently: a row's sums may differ by what each is off"""
    g, K = gen(3), 2048
    a, w = randn(g, 257, K), randn(g, 384, K)
    ref = a.double() @ w.double().T
    rows = [ops.glinear(a[:M], w, out_dtype=F32)[:1] for M in (1, 16, 17, 64, 65, 257)]
    assert torch.equal(rows[0], rows[1]) and torch.equal(rows[2], rows[3]) and torch.equal(rows[4], rows[5])
    for r in rows:
        assert rel(r, ref[:1]) < acc(K) and rel(r, rows[0].double()) < 2 * acc(K)


@pytest.mark.parametrize("routed", [False, True])
@pytest.mark.parametrize("rows", [40, 600])
def test_glinear_waits_that_run_out_are_reported(ops, monkeypatch, rows, routed):
    """waits of 0 tries give up at once, few tries somewhere under way: the launch ends, the next status says so once, and the
    kernel works as before"""
    from vila_b200 import _lib
    g, K, N, E = gen(rows), 1024, 256, 4
    a, w = randn(g, rows, K), randn(g, *((E, N, K) if routed else (N, K)))
    kw = {}
    if routed:
        idx = torch.randint(0, E, (rows, 1), generator=g, device="cuda", dtype=torch.int32)
        seg, srt = ops.moe_group(idx, E)
        kw = dict(groups=E, seg=seg, a_rows=srt, a_row_div=1)
    lib = _lib.load()
    before = lib.vila_stalled_waits()

    def limited(tries):
        out = torch.full((rows, N), 7.0, device="cuda")
        with monkeypatch.context() as m:
            m.setattr(lib, "vila_glinear", lambda p, stream: lib.vila_glinear_tries(p, tries, stream))
            ops.glinear(a, w, out=out, **kw)
        torch.cuda.synchronize()
        return out

    want = limited(1 << 20)
    ops.check_waits()
    assert rel(want, ops.glinear(a, w, out_dtype=F32, **kw).double()) < acc(K)
    for tries in (0, 1, 3, 30):
        out = limited(tries)
        if tries == 0 or not torch.equal(out, want):
            with pytest.raises(RuntimeError, match="ran out"):
                ops.check_waits()
        else:
            lib.vila_wait_status()
        ops.check_waits()
    assert lib.vila_stalled_waits() > before
    limited(0)
    with pytest.raises(RuntimeError, match="ran out"):
        ops.glinear(a, w, out_dtype=F32, **kw)     # the next call says so as well
    limited(0)
    from vila_b200.serving import TokenEngine
    with pytest.raises(RuntimeError, match="ran out"):
        TokenEngine.step(object.__new__(TokenEngine), [])   # and the engine before it builds a step on that output
    assert torch.equal(limited(1 << 20), want)


@pytest.mark.parametrize("role", [0, 1, 2, 3])
@pytest.mark.parametrize("rows,routed", [(40, False), (9, True), (200, True), (600, True), (600, False)])
def test_glinear_gives_up_behind_work_in_flight(ops, rows, routed, role):
    """one role of the CTAs gives up at its first wait while the others' waits hold: tiles that are still landing and products behind
    which nobody looks are drained all the same; the launch ends and the next ones are right.  K of fewer stages than the ring has"""
    from vila_b200 import _lib
    lib, g, N, E = _lib.load(), gen(rows + role), 300, 4
    if role == 2 and not routed:
        return   # no rows are gathered
    for K in (128, 1024):
        a, w, kw = randn(g, rows, K), randn(g, *((E, N, K) if routed else (N, K))), {}
        if routed:
            seg, srt = ops.moe_group(torch.randint(0, E, (rows, 1), generator=g, device="cuda", dtype=torch.int32), E)
            kw = dict(groups=E, seg=seg, a_rows=srt, a_row_div=1)

        def limited(tries):
            with pytest.MonkeyPatch.context() as m:
                m.setattr(lib, "vila_glinear", lambda p, stream: lib.vila_glinear_tries(p, tries, stream))
                out = ops.glinear(a, w, out_dtype=F32, **kw)
            torch.cuda.synchronize()
            return out

        want = limited(1 << 20)
        ops.check_waits()
        for _ in range(3):
            limited(-2 - role)
            with pytest.raises(RuntimeError, match="ran out"):
                ops.check_waits()
            assert torch.equal(limited(1 << 20), want)
    ops.check_waits()


def test_engine_reports_a_step_that_gave_up_before_a_second_one_builds_on_it(ops):
    """a step whose logits nobody reads gives up behind a second of other work: the step after next raises"""
    from vila_b200 import _lib
    from vila_b200.serving import TokenEngine
    lib, g = _lib.load(), gen(1)
    a, w = randn(g, 64, 256), randn(g, 256, 256)

    class Model:
        device, dtype, tries = torch.device("cuda", torch.cuda.current_device()), BF, 1 << 20
        latent_widths = state_shapes = staticmethod(dict)

        def forward_step(self, batch, cache, layer_outputs=None):
            if self.tries == 0:
                torch.cuda._sleep(2_000_000_000)
                with pytest.MonkeyPatch.context() as m:
                    m.setattr(lib, "vila_glinear", lambda p, stream: lib.vila_glinear_tries(p, 0, stream))
                    ops.glinear(a, w)
            return a

    ops.check_waits()
    model = Model()
    engine = TokenEngine(model, 256, 1, graphs=False)
    engine.step([(0, [1, 2, 3], [])])
    model.tries = 0
    engine.step([(0, [4], [])])
    model.tries = 1 << 20
    engine.step([(0, [5], [])])
    try:
        with pytest.raises(RuntimeError, match="ran out"):
            engine.step([(0, [6], [])])
    finally:
        torch.cuda.synchronize()
        lib.vila_wait_status()
    assert engine.length(0) == 5
    engine.step([(0, [6], [])])
    ops.check_waits()


@pytest.mark.parametrize("pairs,E", [(1, 1), (31, 5), (256, 32), (257, 7), (8192, 32), (8191, 300), (20000, 64), (600, 1500), (9000, 1100)])
def test_moe_group_is_a_stable_sort(ops, pairs, E):
    """expert segments in pair order; indices of no expert (identity choices) belong to no segment"""
    g = gen(pairs)
    idx = torch.randint(0, E + 3, (pairs,), generator=g, device="cuda", dtype=torch.int32)
    seg, srt = ops.moe_group(idx, E)
    want = [torch.nonzero(idx == e).view(-1) for e in range(E)]
    assert seg.tolist() == [0] + torch.tensor([w.numel() for w in want]).cumsum(0).tolist()
    assert torch.equal(srt[:int(seg[-1])].long(), torch.cat(want))


@pytest.mark.parametrize("pairs", [257, 512, 2049, 8192, 8193])
@pytest.mark.parametrize("E", [1, 4, 63, 64, 65, 128, 256, 4096])
def test_moe_group_at_the_ends_of_its_forms(ops, pairs, E):
    """scanned and walked counts, lanes kept and found again, one to 32 warps, tables that just fit shared memory and do not"""
    idx = torch.randint(-1, E + 1, (pairs,), generator=gen(pairs + E), device="cuda", dtype=torch.int32)
    seg, srt = ops.moe_group(idx, E)
    order = torch.argsort(torch.where((idx >= 0) & (idx < E), idx, E), stable=True)
    n = torch.bincount(idx[(idx >= 0) & (idx < E)].long(), minlength=E)
    assert torch.equal(seg[1:].long(), n.cumsum(0)) and int(seg[0]) == 0
    assert torch.equal(srt[:int(seg[-1])].long(), order[:int(seg[-1])])


@pytest.mark.parametrize("rows", [1, 256, 257, 1184, 1191])
@pytest.mark.parametrize("cols", [256, 1030])
def test_moe_route_forms_agree(ops, rows, cols):
    """however many tokens and outputs a CTA takes, a token's choice and weights are the same bits"""
    g = gen(rows)
    x, w, c = randn(g, rows, cols), randn(g, 37, cols, dtype=F32) * cols ** -0.5, randn(g, 36, dtype=F32) * 0.05
    kw = dict(score=ops.SCORE_SOFTMAX, groups=4, keep=2, group_top=2, scale=2.0, gate_w=w[36].contiguous())
    idx, wt, gate = ops.moe_route_scores(x, w[:36].contiguous(), c, 5, **kw)
    for r in sorted({0, rows // 2, rows - 1}):
        one = ops.moe_route_scores(x[r:r + 1].contiguous(), w[:36].contiguous(), c, 5, **kw)
        assert torch.equal(one[0][0], idx[r]) and torch.equal(one[1][0], wt[r]) and torch.equal(one[2][0], gate[r])


@pytest.mark.parametrize("rows,cols,pad", [(1184, 4, 4), (1200, 132, 4), (1185, 1028, 12), (1191, 2048, 0)])
@pytest.mark.parametrize("E,groups", [(8, 2), (32, 4), (33, 3), (100, 5)])
def test_moe_route_tiles_give_the_bits_of_one_token(ops, rows, cols, pad, E, groups):
    """tiles of 16 tokens x 32 experts x 128 columns, the last ones in part: choice and weights of a token alone"""
    g = gen(rows + E)
    x, w, c = randn(g, rows, cols + pad)[:, :cols], randn(g, E, cols, dtype=F32) * cols ** -0.5, randn(g, E, dtype=F32) * 0.05
    idx, wt = ops.moe_route_sigmoid(x, w, c, 3, groups, 2)
    for r in sorted({0, 15, 16, rows // 2, rows - 2, rows - 1}):
        one = ops.moe_route_sigmoid(x[r:r + 1].contiguous(), w, c, 3, groups, 2)
        assert torch.equal(one[0][0], idx[r]) and torch.equal(one[1][0], wt[r])


@pytest.mark.parametrize("rows,cols,E,groups", [(1185, 2048, 32, 4), (2049, 1028, 64, 4), (1200, 4096, 128, 8), (3601, 132, 33, 3), (2368, 64, 97, 1)])
def test_moe_route_tiles_of_many_tokens(ops, rows, cols, E, groups):
    """sizes that go to tiles of 16 tokens x 32 experts whichever number of SMs up to 148 holds them: the bits of a token alone"""
    g = gen(rows)
    x, w, c = randn(g, rows, cols + (-cols) % 8)[:, :cols], randn(g, E, cols, dtype=F32) * cols ** -0.5, randn(g, E, dtype=F32) * 0.05
    idx, wt = ops.moe_route_sigmoid(x, w, c, 3, groups, max(1, groups // 2))
    for r in sorted({0, 15, 16, rows // 2, rows - 2, rows - 1}):
        one = ops.moe_route_sigmoid(x[r:r + 1].contiguous(), w, c, 3, groups, max(1, groups // 2))
        assert torch.equal(one[0][0], idx[r]) and torch.equal(one[1][0], wt[r])


@pytest.mark.parametrize("rows,cols,np_", [(1, 4, 1), (3, 1028, 2), (300, 2048, 4), (5, 136, 7)])
@pytest.mark.parametrize("a_dt", [None, BF, F32])
def test_residual_add_vec_equals_the_general_form(ops, rows, cols, np_, a_dt):
    """four columns a thread against one: the same sums in the same order (the general form is forced by an odd stride)"""
    g = gen(rows + np_)
    x, part = randn(g, rows, cols, dtype=F32), randn(g, rows * np_, cols + 1, dtype=F32)[:, :cols]
    a = None if a_dt is None else randn(g, rows, cols, dtype=a_dt)
    y = x.clone()
    c0 = ops.residual_add_rows(x, a, part, n_partials=np_, mult=0.5, copy_dtype=BF)
    c1 = ops.residual_add_rows(y, a, part.contiguous(), n_partials=np_, mult=0.5, copy_dtype=BF)
    assert torch.equal(x, y) and torch.equal(c0, c1)


# ---- paged attention of prompt portions ---------------------------------------------------------------------
ATT_FORMS = {"plain": {}, "capped": dict(softcap=5.0, gate=True), "sink": dict(sink=True, head_scale=True), "window": dict(window=21, keep_first=3),
             "narrow": dict(window=5, gate=True), "chunk": dict(chunk=24, dist_bias=30, sink=True, gate=True),
             "diff": dict(diff=(0.4, 0.6, 1e-5), window=37, gate=True), "diff_plain": dict(diff=(0.3, 0.7, 1e-5))}


def attention_reference(q, pool, tables, seqs, H, G, D, V, page, scale, o):
    """float64, row by row of positions; seqs: (row0, rows, pos0, slot)"""
    maps = 2 if "diff" in o else 1
    out = torch.empty(q.shape[0], H, V, device="cuda", dtype=torch.float64)
    for row0, n, pos0, slot in seqs:
        j = torch.arange(pos0 + n, device="cuda")
        rows = tables[slot, j // page].long() * page + j % page
        k, v = pool[rows, :G * maps * D].double().view(-1, G, maps, D), pool[rows, G * maps * D:].double().view(-1, G, V)
        i = pos0 + torch.arange(n, device="cuda")
        back = i[:, None] - j[None]
        see = back >= 0
        if "window" in o:
            see &= (back < o["window"]) | (j[None] < o.get("keep_first", 0))
        if "chunk" in o:
            see &= j[None] >= (i[:, None] // o["chunk"]) * o["chunk"]
        s = torch.einsum("ihmd,jhmd->hmij", q[row0:row0 + n].double().view(n, H, maps, D), k.repeat_interleave(H // G, 1)) * scale
        if "head_scale" in o:
            s = s * o["head_scale"].double()[:, None, None, None]
        if "softcap" in o:
            s = o["softcap"] * torch.tanh(s / o["softcap"])
        if "talk" in o and not o.get("talk_after"):
            s = torch.einsum("hg,gmij->hmij", o["talk"].double(), s)
        if "dist_bias" in o:
            s = s + o["dist_bias"].double()[back.clamp(0, o["dist_bias"].shape[0] - 1)].permute(2, 0, 1)[:, None]
        s = s.masked_fill(~see, float("-inf"))
        if "sink" in o:
            s = torch.cat([s, o["sink"].double()[:, None, None, None].expand(H, maps, n, 1)], -1)
        w = torch.softmax(s, -1)[..., :pos0 + n]
        if o.get("talk_after"):
            w = torch.einsum("hg,gmij->hmij", o["talk"].double(), w)
        a = torch.einsum("hmij,jhd->ihmd", w, v.repeat_interleave(H // G, 1))
        if maps == 2:
            lam, sc, eps = o["diff"]
            a = a[:, :, 0] - lam * a[:, :, 1]
            a = a / torch.sqrt(a.pow(2).mean(-1, keepdim=True) + eps) * sc
        else:
            a = a[:, :, 0]
        if "gate" in o:
            a = a * torch.sigmoid(o["gate"][row0:row0 + n].double())[..., None]
        out[row0:row0 + n] = a
    return out.view(q.shape[0], -1)


def attention_case(ops, form, H, G, D, V, page, seqs, seed, q_scale=1.0, scale=0.1, **call):
    g, o = gen(seed), dict(form)
    maps = 2 if "diff" in o else 1
    T, slots = sum(n for n, _ in seqs), len(seqs)
    pages = max((p + n + page - 1) // page for n, p in seqs)
    pool = randn(g, slots * pages * page, G * (maps * D + V))
    tables = torch.randperm(slots * pages, generator=g, device="cuda").to(torch.int32).view(slots, pages)
    q = torch.randn(T, H * maps * D, generator=g, device="cuda") * q_scale
    for k, shape in (("gate", (T, H)), ("sink", (H,)), ("head_scale", (H,))):
        if o.get(k) is True:
            o[k] = torch.randn(shape, generator=g, device="cuda") * 0.5 + (1.0 if k == "head_scale" else 0.0)
    if isinstance(o.get("dist_bias"), int):
        o["dist_bias"] = torch.randn(o["dist_bias"], H, generator=g, device="cuda")
    if o.get("talk") is True:
        o["talk"] = torch.eye(H, device="cuda") + 0.3 * torch.randn(H, H, generator=g, device="cuda")
    at, spans = 0, []
    for s, (n, p) in enumerate(seqs):
        spans.append((at, n, p, s))
        at += n
    step = call.get("max_rows", 16)
    tiles = torch.tensor([(r + i, min(step, n - i), p + i, s) for r, n, p, s in spans for i in range(0, n, step)], dtype=torch.int32, device="cuda")
    call.setdefault("max_rows", 16)
    got = ops.paged_attention(q, pool, tables, tiles, heads=H, kv_heads=G, dim=D, vdim=V, page=page, scale=scale, out_dtype=F32, **call, **o)
    return got, attention_reference(q, pool, tables, spans, H, G, D, V, page, scale, o), (q, pool, tables, tiles, o)


@pytest.mark.parametrize("form", list(ATT_FORMS))
@pytest.mark.parametrize("rep", [1, 2, 3, 4, 5, 8])
@pytest.mark.parametrize("seqs", [[(2, 0)], [(16, 0), (17, 63), (3, 128)], [(200, 0)], [(33, 300), (64, 1)]])
def test_paged_attention_prompt(ops, form, rep, seqs):
    """fp32 results of bf16 caches: a score sums 128 products of three parts, a row up to 333 weights; 3e-6 of the norm.
    Capped, biased and masked forms, tiles of 1 to 16 rows, several sequences in one launch, page sizes 16 and 64."""
    o = ATT_FORMS[form]
    D, V = (64, 128) if "diff" in o else (128, 128)
    if "diff" in o and rep > 4:
        rep = 4   # eight score heads of a key head
    got, want, _ = attention_case(ops, o, 2 * rep, 2, D, V, 16 if rep % 2 else 64, seqs, seed=rep)
    assert rel(got, want) < 3e-6
    if form == "plain":
        got, want, _ = attention_case(ops, o, 2 * rep, 2, 64, 64, 48, seqs, seed=rep)
        assert rel(got, want) < 3e-6


def test_paged_attention_prompt_extremes(ops):
    """large scores (one key takes a row), and a row whose result does not depend on what else is in the launch"""
    got, want, (q, pool, tables, tiles, o) = attention_case(ops, {}, 8, 2, 128, 128, 64, [(40, 90), (25, 0)], seed=5, q_scale=30.0, scale=1.0)
    assert torch.isfinite(got).all() and rel(got, want) < 1e-4   # scores of several hundred: their last bits are 3e-5 of a weight
    kw = dict(heads=8, kv_heads=2, dim=128, vdim=128, page=64, scale=1.0, out_dtype=F32, max_rows=16)
    alone = ops.paged_attention(q, pool, tables, tiles[1:2].contiguous(), **kw)
    assert torch.equal(alone[16:32], got[16:32])
    q[3, 7] = float("nan")
    assert torch.isnan(ops.paged_attention(q, pool, tables, tiles, **kw)[3, :128]).all()


@pytest.mark.parametrize("cap", [0.01, 1.0, 11.3, 1e9])
@pytest.mark.parametrize("max_rows,talk", [(16, False), (1, False), (16, True)])
def test_paged_attention_scores_around_the_cap(ops, cap, max_rows, talk):
    """scores far below the cap, next to it (where tanh changes its form) and above it; the same bits wherever a tile begins"""
    form = dict(softcap=cap, **(dict(talk=True) if talk else {}))
    got, want, (q, pool, tables, tiles, o) = attention_case(ops, form, 8, 2, 128, 128, 64, [(70, 30)], seed=3, scale=0.3, max_rows=max_rows)
    assert rel(got, want) < 3e-6
    if max_rows == 16 and not talk:
        kw = dict(heads=8, kv_heads=2, dim=128, vdim=128, page=64, scale=0.3, out_dtype=F32, max_rows=16, **o)
        other = torch.tensor([(r, min(16, 70 - r), 30 + r, 0) for r in range(5, 70, 16)], dtype=torch.int32, device="cuda")
        assert torch.equal(ops.paged_attention(q, pool, tables, other, **kw)[5:], got[5:])


@pytest.mark.parametrize("max_rows,talk", [(16, False), (1, False), (16, True)])
def test_paged_attention_scores_far_above_the_cap(ops, max_rows, talk):
    """scores whose exponential is infinite are the cap itself"""
    form = dict(softcap=5.0, **(dict(talk=True) if talk else {}))
    got, want, _ = attention_case(ops, form, 8, 2, 128, 128, 64, [(40, 30)], seed=4, scale=1e25, max_rows=max_rows)
    assert torch.isfinite(got).all() and rel(got, want) < 3e-6


@pytest.mark.parametrize("max_rows,nsplit", [(16, 1), (1, 1), (1, 8)])
def test_paged_attention_sink_switched_off(ops, max_rows, nsplit):
    """a sink of -inf (or below every score) adds nothing to a head's sum; the other heads keep theirs"""
    sink = torch.tensor([float("-inf"), 0.5, -2e30, 1.5], device="cuda")
    seqs = [(40, 90), (17, 0)] if max_rows > 1 else [(1, 130), (1, 0)]
    got, want, _ = attention_case(ops, {"sink": sink}, 4, 2, 128, 128, 64, seqs, seed=9, max_rows=max_rows, nsplit=nsplit)
    assert rel(got, want) < 3e-6


@pytest.mark.parametrize("keys", [64, 333, 2048, 4096, 16384])
@pytest.mark.parametrize("D,G", [(64, 2), (128, 2), (128, 8)])
def test_paged_attention_prompt_long(ops, keys, D, G):
    """the error does not grow with the keys as it would in one truncating sum (8e-6 at 2048 keys): 32 keys are summed on
    the tensor core, two truncations of that size, and the keys / 32 parts by rounded additions, whose errors go both ways"""
    got, want, _ = attention_case(ops, {}, 8, G, D, D, 64, [(40, keys - 40)], seed=keys, scale=0.05)
    assert rel(got, want) < 4e-7 + (keys / 32) ** 0.5 * 2.0 ** -25


@pytest.mark.parametrize("form", ["plain", "capped", "window", "chunk", "diff_plain"])
@pytest.mark.parametrize("rep", [1, 4, 8])
def test_paged_attention_prompt_infinite_entries(ops, form, rep):
    """an infinite value reaches the rows that see it and nothing else (earlier rows of its tile and of its CTA keep their
    numbers); a score of -inf weighs nothing"""
    o, H = ATT_FORMS[form], 2 * min(rep, 4 if "diff" in ATT_FORMS[form] else 8)
    D, V, maps, page, T, j = (64, 128, 2, 64, 90, 37) if "diff" in o else (128, 128, 1, 64, 90, 37)
    got, want, (q, pool, tables, tiles, o) = attention_case(ops, o, H, 2, D, V, page, [(T, 0)], seed=rep)
    kw = dict(heads=H, kv_heads=2, dim=D, vdim=V, page=page, scale=0.1, out_dtype=F32, max_rows=16, **o)
    row = int(tables[0, j // page]) * page + j % page
    bad = pool.clone()
    bad[row, 2 * maps * D + 5] = float("inf")                       # value column 5 of the first key head
    inf = ops.paged_attention(q, bad, tables, tiles, **kw)
    assert rel(inf[:j], want[:j]) < 3e-6
    heads = inf.view(T, H, V)[:, :H // 2]                           # of that key head
    assert rel(inf.view(T, H, V)[:, H // 2:], want.view(T, H, V)[:, H // 2:]) < 3e-6
    reach = min(T, j + o.get("window", T), (j // o["chunk"] + 1) * o["chunk"] if "chunk" in o else T)
    if "diff" in o:
        assert not torch.isfinite(heads[j:reach, :, 5]).any()       # inf - lambda inf
    else:
        assert torch.isinf(heads[j:reach, :, 5]).all()
        others = [c for c in range(V) if c != 5]
        assert rel(heads[:, :, others], want.view(T, H, V)[:, :H // 2][:, :, others]) < 3e-6
        q = q.clone()
        q.view(T, H, D)[:, :, 3] = q.view(T, H, D)[:, :, 3].abs() + 0.1
        bad = pool.clone()
        bad[row, 3] = float("-inf")
        if "softcap" not in o:                                      # a capped score is finite
            ref = attention_reference(q, bad, tables, [(0, T, 0, 0)], H, 2, D, V, page, 0.1, o)
            got = ops.paged_attention(q, bad, tables, tiles, **kw)
            seen = torch.isfinite(ref).all(1)                       # (a row that sees no other key has no number)
            assert int(seen.sum()) > T - 3 and rel(got[seen], ref[seen]) < 3e-6


@pytest.mark.parametrize("tries", [0, 1, 3, 30, -2, -3, -4])
@pytest.mark.parametrize("seqs", [[(9, 0)], [(40, 300), (64, 1)], [(200, 0)]])
def test_paged_attention_prompt_waits_that_run_out(ops, tries, seqs):
    """all waits give up at once or somewhere under way, or (negative) those of one role do while the others' hold, so that products
    are in flight behind which nobody looks: the launch ends, the next status says so once, and the kernel works as before"""
    from vila_b200 import _lib
    lib = _lib.load()
    for form in (dict(softcap=30.0, gate=True), dict(dist_bias=11, chunk=100)):
        want, ref, (q, pool, tables, tiles, o) = attention_case(ops, form, 8, 2, 128, 128, 64, seqs, seed=3)
        kw = dict(heads=8, kv_heads=2, dim=128, vdim=128, page=64, scale=0.1, out_dtype=F32, max_rows=16, **o)
        assert rel(want, ref) < 3e-6
        ops.check_waits()
        for _ in range(3):
            with pytest.MonkeyPatch.context() as m:
                m.setattr(lib, "vila_paged_attention", lambda p, stream: lib.vila_paged_attention_tries(p, tries, stream))
                out = ops.paged_attention(q, pool, tables, tiles, **kw)
            torch.cuda.synchronize()
            if tries <= 0 or not torch.equal(out, want):
                with pytest.raises(RuntimeError, match="ran out"):
                    ops.check_waits()
            else:
                lib.vila_wait_status()
            assert torch.equal(ops.paged_attention(q, pool, tables, tiles, **kw), want)
    ops.check_waits()


def test_paged_attention_prompt_refuses_to_build_on_a_launch_that_gave_up(ops):
    """a prompt's attention behind an incomplete one, or behind an incomplete linear layer, raises before it launches anything"""
    from vila_b200 import _lib
    lib, g = _lib.load(), gen(2)
    want, _, (q, pool, tables, tiles, o) = attention_case(ops, {}, 8, 2, 128, 128, 64, [(40, 30)], seed=2)
    kw = dict(heads=8, kv_heads=2, dim=128, vdim=128, page=64, scale=0.1, out_dtype=F32, max_rows=16)
    a, w = randn(g, 40, 256), randn(g, 256, 256)
    for name, call in (("vila_paged_attention", lambda: ops.paged_attention(q, pool, tables, tiles, **kw)), ("vila_glinear", lambda: ops.glinear(a, w))):
        with pytest.MonkeyPatch.context() as m:
            m.setattr(lib, name, lambda p, stream: getattr(lib, name + "_tries")(p, 0, stream))
            call()
        torch.cuda.synchronize()
        with pytest.raises(RuntimeError, match="vila_paged_attention.*ran out"):
            ops.paged_attention(q, pool, tables, tiles, **kw)
        assert torch.equal(ops.paged_attention(q, pool, tables, tiles, **kw), want)
    ops.check_waits()


@pytest.mark.parametrize("rows", [1900, 2100])
def test_paged_attention_prompt_bias_of_many_distances(ops, rows):
    """tables by distance that just fit beside the operands in shared memory and that do not; distances past their end"""
    for seqs in ([(33, 300), (64, 1)], [(20, 2300)]):
        got, want, _ = attention_case(ops, dict(dist_bias=rows, gate=True), 8, 2, 128, 128, 64, seqs, seed=rows)
        assert rel(got, want) < 3e-6


@pytest.mark.parametrize("form", [dict(), dict(softcap=5.0, sink=True), dict(window=300, keep_first=70), dict(window=90, keep_first=130, dist_bias=40), dict(chunk=200, dist_bias=250)])
@pytest.mark.parametrize("H,G", [(32, 32), (12, 4), (32, 8), (16, 2)])
def test_paged_attention_prompt_rows_do_not_depend_on_their_cta(ops, form, H, G):
    """tiles of several sequences and positions side by side in a CTA, whose other rows see other blocks, against launches of one
    tile: the same bits, and CTAs of one tile (few rows, heads that do not divide 8) are as right as full ones"""
    seqs = [(16, 700), (40, 0), (3, 900), (64, 500), (1, 65), (17, 250), (33, 1000), (2, 0), (50, 333), (5, 64)] * (2 if G < 8 else 1)
    got, want, (q, pool, tables, tiles, o) = attention_case(ops, form, H, G, 128, 128, 64, seqs, seed=H)
    assert rel(got, want) < 3e-6
    for t in tiles:
        r0, n = int(t[0]), int(t[1])
        alone = ops.paged_attention(q, pool, tables, t[None].contiguous(), heads=H, kv_heads=G, dim=128, vdim=128, page=64, scale=0.1, out_dtype=F32,
                                    max_rows=16, **o)
        assert torch.equal(alone[r0:r0 + n], got[r0:r0 + n])


@pytest.mark.parametrize("keys", [64, 128, 192, 256, 512, 704, 2048, 3008])
@pytest.mark.parametrize("form", ["signs", "one", "chunk"])
def test_paged_attention_prompt_error_does_not_grow_with_the_keys(ops, keys, form):
    """rounding of fp32 sums over up to 3008 keys.  Values of one sign: a block's four truncated additions of 16 weights' first
    parts are 2^-24 each of what they add to, half that on average and all one way (0.8e-7), a row's value is rounded once (0.3e-7
    rms) and its quotient once; 1.2e-7 holds them, while a plain sum of the blocks adds 1e-8 sqrt(blocks) and is past it from 1000
    keys on.  Both signs: the weights' own error, of scores whose 128 products are added in two sums of 64, on top: 2.4e-7"""
    e = []
    for seed in range(6):
        g, R, H, G, D = gen(seed), 64, 16, 4, 128
        q, kv = torch.randn(R, H * D, generator=g, device="cuda"), torch.randn(keys, 2 * G * D, generator=g, device="cuda")
        if form != "signs":
            kv[:, G * D:] = kv[:, G * D:].abs()
        pool, o = kv.to(BF), dict(chunk=512) if form == "chunk" else {}
        tables = torch.arange(keys // 64, dtype=torch.int32, device="cuda")[None].contiguous()
        tiles = torch.tensor([(r, 16, keys - R + r, 0) for r in range(0, R, 16)], dtype=torch.int32, device="cuda")
        got = ops.paged_attention(q, pool, tables, tiles, heads=H, kv_heads=G, dim=D, vdim=D, page=64, scale=D ** -0.5, out_dtype=F32, max_rows=16, **o)
        want = attention_reference(q, pool, tables, [(0, R, keys - R, 0)], H, G, D, D, 64, D ** -0.5, o)
        e.append(rel(got, want))
    assert sum(e) / len(e) < (2.4e-7 if form == "signs" else 1.2e-7)


MIX_FORMS = {"talk": dict(talk=True), "sink": dict(talk=True, sink=True, softcap=5.0, gate=True), "chunk": dict(talk=True, chunk=24, dist_bias=30),
             "after": dict(talk=True, talk_after=True), "after_window": dict(talk=True, talk_after=True, window=21, keep_first=3, head_scale=True, gate=True)}


@pytest.mark.parametrize("form", list(MIX_FORMS))
@pytest.mark.parametrize("H,G", [(2, 1), (7, 7), (8, 2), (16, 4), (17, 17), (32, 32), (32, 8)])
@pytest.mark.parametrize("seqs", [[(2, 0)], [(16, 0), (17, 63), (3, 128)], [(33, 300), (64, 1)]])
def test_paged_attention_prompt_mixed_heads(ops, form, H, G, seqs):
    """a mixed score (weight) is a sum over H heads of mean square 1 + 0.09 H: the 3e-6 of one head times its root, at most 6e-6;
    tiles of 1 to 16 rows, one and two heads a warp, warps without a head, rows alone"""
    for D in (64, 128):
        got, want, (q, pool, tables, tiles, o) = attention_case(ops, MIX_FORMS[form], H, G, D, D, 48 if H == 8 else 64, seqs, seed=H)
        assert rel(got, want) < 6e-6
        one = torch.stack([tiles[-1, 0] + tiles[-1, 1] - 1, torch.ones_like(tiles[-1, 0]), tiles[-1, 2] + tiles[-1, 1] - 1, tiles[-1, 3]])[None].contiguous()
        alone = ops.paged_attention(q, pool, tables, one, heads=H, kv_heads=G, dim=D, vdim=D, page=48 if H == 8 else 64, scale=0.1, out_dtype=F32,
                                    max_rows=16, **o)
        assert torch.equal(alone[-1], got[-1])


@pytest.mark.parametrize("form", list(MIX_FORMS))
@pytest.mark.parametrize("H", [4, 20])
def test_paged_attention_prompt_mixed_heads_infinite_value(ops, form, H):
    """an infinite value reaches the rows that see it (all heads of its value head) and nothing else"""
    T, j, D, o = 70, 37, 128, MIX_FORMS[form]
    got, want, (q, pool, tables, tiles, o) = attention_case(ops, o, H, H // 2, D, D, 64, [(T, 0)], seed=H)
    bad = pool.clone()
    bad[int(tables[0, j // 64]) * 64 + j % 64, H // 2 * D + 5] = float("inf")
    inf = ops.paged_attention(q, bad, tables, tiles, heads=H, kv_heads=H // 2, dim=D, vdim=D, page=64, scale=0.1, out_dtype=F32, max_rows=16, **o).view(T, H, D)
    want, reach = want.view(T, H, D), min(T, j + o.get("window", T), (j // o["chunk"] + 1) * o["chunk"] if "chunk" in o else T)
    assert torch.isinf(inf[j:reach, :2, 5]).all()
    keep = torch.ones_like(want, dtype=torch.bool)
    keep[j:reach, :2, 5] = False
    assert torch.isfinite(inf[keep]).all() and rel(inf[keep], want[keep]) < 6e-6


def test_paged_attention_decode_skips_empty_tiles(ops):
    """a tile of no rows names an output row but has nothing to write"""
    for nsplit in (1, 4):
        got, _, (q, pool, tables, tiles, o) = attention_case(ops, {}, 8, 2, 128, 128, 64, [(1, 100), (1, 30), (1, 5)], seed=2, max_rows=1, nsplit=nsplit)
        tiles = tiles.clone()
        tiles[1, 1] = 0
        out = torch.full_like(got, 7.0)
        ops.paged_attention(q, pool, tables, tiles, heads=8, kv_heads=2, dim=128, vdim=128, page=64, scale=0.1, max_rows=1, nsplit=nsplit, out=out)
        assert bool((out[1] == 7.0).all()) and torch.equal(out[0], got[0]) and torch.equal(out[2], got[2])


@pytest.mark.parametrize("dim,rot,halves,H,dtype,pool_dtype", [(64, 64, True, 5, BF, BF), (128, 40, False, 3, F32, BF), (128, 56, True, 4, BF, F32),
                                                               (256, 256, False, 2, BF, BF)])
@pytest.mark.parametrize("k_values", [False, True])
def test_rope_append_tokens_of_a_cta(ops, dim, rot, halves, H, dtype, pool_dtype, k_values):
    """two tokens per CTA and a last one with one: the bits of one per CTA, and within rounding of rows that start off 8 bytes"""
    T = 4 * torch.cuda.get_device_properties(0).multi_processor_count + 3
    g, G = gen(dim), 2
    V = dim if k_values else 20
    n = (H + G) * dim + (0 if k_values else G * V)
    qkv = randn(g, T, n, dtype=dtype)
    off = torch.cat([qkv.new_zeros(1), qkv.flatten()])[1:].view(T, n)
    pos, rows = (torch.randperm(T, generator=g, device="cuda").int() for _ in range(2))
    inv = 10000.0 ** (-2.0 * torch.arange(rot // 2, device="cuda", dtype=torch.float64) / rot)
    out = []
    for x, step in ((qkv, T), (qkv, 100), (off, T)):
        pool, q = torch.zeros(T, G * (dim + V), device="cuda", dtype=pool_dtype), []
        for t in range(0, T, step):
            s = slice(t, t + step)
            q.append(ops.rope_append(x[s], pos[s].contiguous(), rows[s].contiguous(), pool, heads=H, kv_heads=G, dim=dim, vdim=V, inv_freq=inv,
                                     unit_norm=True, eps=1e-5, halves=halves, v_from_k=k_values))
        out.append((torch.cat(q), pool))
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
    # fp32: the norm's sum of dim squares in another order; bf16: one step of rounding
    assert rel(out[0][0], out[2][0].double()) < 5e-7 and rel(out[0][1], out[2][1].double()) < (5e-7 if pool_dtype == F32 else 2 ** -7)


@pytest.mark.parametrize("dim,rot,halves", [(2, 2, False), (64, 64, True), (96, 32, False), (128, 64, True), (130, 128, False), (256, 256, True)])
@pytest.mark.parametrize("dtype", [BF, F32])
def test_rope_append_pairs(ops, dim, rot, halves, dtype):
    """a lane's pairs of columns at head sizes below, at and past its 32: against float64 angles, unit norm with weights, value mixing"""
    g, T, H, G, V = gen(dim), 5, 3, 2, 24
    qkv, vf = randn(g, T, (H + G) * dim + G * V, dtype=dtype), randn(g, T, G * V, dtype=dtype)
    pos = torch.tensor([0, 1, 77, 5000, 100000], dtype=torch.int32, device="cuda")
    rows, pool = torch.tensor([4, 0, 3, 1, 2], dtype=torch.int32, device="cuda"), torch.zeros(5, G * (dim + V), device="cuda", dtype=F32)
    inv = 10000.0 ** (-2.0 * torch.arange(rot // 2, device="cuda", dtype=torch.float64) / rot)
    w = [1 + 0.1 * torch.randn(dim, generator=g, device="cuda") for _ in range(2)]
    q = ops.rope_append(qkv, pos, rows, pool, heads=H, kv_heads=G, dim=dim, vdim=V, inv_freq=inv, unit_norm=True, eps=1e-5, q_norm_w=w[0],
                        k_norm_w=w[1], halves=halves, mscale=1.25, v_first=vf, v_mix=0.3)
    x = qkv.double()[:, :(H + G) * dim].reshape(T, H + G, dim)
    ang = pos.double()[:, None] * inv
    c, s = 1.25 * torch.cos(ang)[:, None], 1.25 * torch.sin(ang)[:, None]
    i = torch.arange(rot // 2, device="cuda")
    i0, i1 = (i, i + rot // 2) if halves else (2 * i, 2 * i + 1)
    y = x.clone()
    y[..., i0], y[..., i1] = x[..., i0] * c - x[..., i1] * s, x[..., i1] * c + x[..., i0] * s
    y = y / torch.sqrt(y.pow(2).mean(-1, keepdim=True) + 1e-5)
    want_q, want_k = y[:, :H] * w[0].double(), y[:, H:] * w[1].double()
    assert rel(q, want_q.reshape(T, -1)) < 5e-7
    want_v = 0.7 * qkv.double()[:, (H + G) * dim:] + 0.3 * vf.double()
    assert rel(pool[rows.long()], torch.cat([want_k.reshape(T, -1), want_v], 1)) < 5e-7


@pytest.mark.parametrize("form", list(ATT_FORMS))
@pytest.mark.parametrize("rep", [1, 2, 4, 8])
@pytest.mark.parametrize("nsplit", [1, 3, 16])
def test_paged_attention_decode(ops, form, rep, nsplit):
    """one row per sequence: contexts below, at and past a group of 16 keys and past all the warps of a cluster"""
    o = ATT_FORMS[form]
    D = 64 if "diff" in o else 128
    seqs = [(1, p) for p in (0, 15, 16, 130, 1500)]
    got, want, _ = attention_case(ops, o, 2 * rep, 2, D, 128, 64 if rep % 2 else 48, seqs, seed=rep, max_rows=1, nsplit=nsplit)
    assert rel(got, want) < 2e-6


@pytest.mark.parametrize("M", [1, 2, 3, 4, 5, 8])
@pytest.mark.parametrize("N,K", [(8, 8), (40, 264), (64, 1024), (64, 4104), (136, 1032), (1000, 2720), (2560, 3592), (4608, 1288)])
def test_linear_few_rows(ops, M, N, K):
    """weight rows and columns below, at and past a warp's four and a pass's 1024, one, two and four warps to a row; every epilogue; bf16 results: half an ulp,
    one more for every rounding in between, of values of the size of their row's norm"""
    g = gen(M * N + K)
    x, w = randn(g, M, K + 8)[:, :K], (randn(g, N, K).float() * K ** -0.5).to(BF)
    b, res = randn(g, N), randn(g, M, N)
    ref = x.double() @ w.double().T
    bf = lambda t: t.to(BF).double()
    assert rel(ops.linear(x, w, static_w=True), ref) < 2.0 ** -8
    z = bf(ref + b.double())
    assert rel(ops.linear(x, w, b, residual=res), z + res.double()) < 2.0 ** -7
    for act, fn in ((ops.ACT_GELU_TANH, lambda t: torch.nn.functional.gelu(t, approximate="tanh")), (ops.ACT_GELU_ERF, torch.nn.functional.gelu),
                    (ops.ACT_SILU, torch.nn.functional.silu), (ops.ACT_RELU2, lambda t: torch.relu(t) ** 2)):
        assert rel(ops.linear(x, w, b, act=act), fn(z)) < 2.0 ** -7
    assert rel(ops.linear(x, w, b, residual=res[:1].contiguous(), res_row_mod=1), z + res[:1].double()) < 2.0 ** -7
    xi = lambda t: torch.where(t > 0, 0.9 * t * t, 0.4 * (torch.expm1(t) - t)) + 0.5 * t
    assert rel(ops.linear(x, w, b, act=ops.ACT_XIELU, act_params=(0.9, 0.4)), xi(z)) < 2.0 ** -7
    if N % 32 == 0:
        gt, u = ref[:, 0::2], ref[:, 1::2]
        assert rel(ops.linear(x, w, swiglu=True), torch.nn.functional.silu(gt) * u) < 2.0 ** -6
        assert rel(ops.linear(x, w, geglu=True), torch.nn.functional.gelu(gt, approximate="tanh") * u) < 2.0 ** -7
        c = gt.clamp_max(0.5)
        assert rel(ops.linear(x, w, glu_clamp=(1.702, 0.5)), c * torch.sigmoid(1.702 * c) * (u.clamp(-0.5, 0.5) + 1)) < 2.0 ** -7
    most = 8 if N * K <= 6000000 else 4                             # rows that this kernel takes of so many weights
    if M <= most:
        many = ops.linear(torch.cat([x] * 8)[:most].contiguous(), w, static_w=True)
        assert torch.equal(many[:M], ops.linear(x, w, static_w=True))   # a row's result does not depend on how many there are


@pytest.mark.parametrize("M", [1, 3, 4, 5, 8, 9, 100, 128, 200, 250, 300])
@pytest.mark.parametrize("Hq,Hkv,K", [(6, 2, 512), (2, 1, 1288), (16, 2, 2048), (28, 4, 3584)])
def test_linear_qkv_rope_equals_linear_and_rope(ops, M, Hq, Hkv, K):
    """the fused projection against vila_linear + vila_rope_kv_append as they dispatch: the same bits where vila_linear takes
    the swap-AB kernel too; few rows of few weights (another kernel) and rows that fill 128-row tiles (halves of K summed
    apart) are another order of the sums: bf16 values that may be a last place apart"""
    g, D, p0 = gen(M + K), 128, 77
    few = (Hq + 2 * Hkv) * D * K <= (20000000 if M <= 4 else 6000000 if M <= 8 else 0)
    halves = M in (128, 250) and (M + 127) // 128 * (Hq + 2 * Hkv) <= torch.cuda.get_device_properties(0).multi_processor_count // 2
    same = (lambda a, b: rel(a, b.double()) < 2.0 ** -8) if few or halves else torch.equal
    N = (Hq + 2 * Hkv) * D
    x, w, b = randn(g, M, K), (randn(g, N, K).float() * K ** -0.5).to(BF), randn(g, N)
    pos = torch.arange(p0, p0 + M, dtype=torch.int32, device="cuda") * 3 + 5
    inv = (1.0 / (1e6 ** (torch.arange(0, D, 2, dtype=torch.float32) / D))).cuda()
    table = torch.randperm(4, generator=torch.Generator().manual_seed(1)).to(torch.int32).cuda()
    pools = [torch.zeros(4, 128, Hkv, D, dtype=BF, device="cuda") for _ in range(4)]
    ref, tab = ops.linear(x, w, b), ops.rope_table(pos, D, inv)
    plain = ref.clone()
    ops.rope_kv_append(ref, pos, Hq, Hkv, D, inv, pools[0], pools[1], table, p0)
    got = ops.linear_qkv_rope(x, w, b, tab, Hq, Hkv, D, pools[2], pools[3], table, p0)
    assert same(got[:, :Hq * D], ref[:, :Hq * D]) and same(pools[2], pools[0]) and same(pools[3], pools[1])
    ops.rope_kv_append(plain, pos, Hq, Hkv, D, inv)
    assert same(ops.linear_qkv_rope(x, w, b, tab, Hq, Hkv, D), plain)


@pytest.mark.parametrize("M", [16, 32, 33, 100, 200, 300, 384])
@pytest.mark.parametrize("Hq,Hkv,K", [(2, 1, 1288), (16, 2, 2048), (28, 4, 3584)])
def test_linear_qkv_rope_without_a_bias(ops, M, Hq, Hkv, K):
    """the same bits up to 32 rows; from 33 on vila_linear may take tiles, which sum K in another order"""
    g, D = gen(M + K), 128
    N = (Hq + 2 * Hkv) * D
    x, w = randn(g, M, K), (randn(g, N, K).float() * K ** -0.5).to(BF)
    pos = torch.arange(M, dtype=torch.int32, device="cuda")
    inv = (1.0 / (1e6 ** (torch.arange(0, D, 2, dtype=torch.float32) / D))).cuda()
    ref, tab = ops.linear(x, w), ops.rope_table(pos, D, inv)
    ops.rope_kv_append(ref, pos, Hq, Hkv, D, inv)
    got = ops.linear_qkv_rope(x, w, None, tab, Hq, Hkv, D)
    assert torch.equal(got, ref) if M <= 32 else rel(got, ref.double()) < 2.0 ** -8


@pytest.mark.parametrize("M,N,K,act,form", [(256, 3584, 4608, 1, 5128), (256, 2048, 4608, 1, 5128), (100, 3584, 4608, 2, 5128), (17, 3584, 4608, 2, 3000), (279, 3584, 18944, 0, 3000),
                                            (64, 2048, 2048, 0, 5128), (32, 2048, 2048, 0, 3000), (384, 1024, 1024, 0, 5128)])
def test_linear_few_tokens_take_the_form_that_is_ahead(ops, M, N, K, act, form):
    """which form vila_linear takes up to 384 rows, by its bits: K summed in order, in the halves of a CTA pair or by a cluster"""
    g = gen(M + N)
    x, w = randn(g, M, K), (randn(g, N, K).float() * K ** -0.5).to(BF)
    got = ops.linear(x, w, act=act)
    others = [f for f in (128, 3000, 5128) if f != form and (f != 5128 or (M + 127) // 128 * ((N + 127) // 128) <= 74)]
    assert torch.equal(got, ops.linear(x, w, act=act, block_n=form)) and not any(torch.equal(got, ops.linear(x, w, act=act, block_n=f)) for f in others)


# ---- recurrences --------------------------------------------------------------------------------------------
def hgrn2_inputs(g, T, H, dim, vdim, dtype=BF):
    proj = randn(g, T, 2 * H * dim + H * vdim, dtype=dtype)
    kw = dict(heads=H, dim=dim, vdim=vdim, q_off=0, f_off=H * dim, v_off=2 * H * dim, f_bias=torch.randn(H * dim, generator=g, device="cuda"),
              lower=torch.rand(H * dim, generator=g, device="cuda") * 0.9)
    q = torch.nn.functional.silu(proj[:, :H * dim].double()).view(T, H, dim)
    low = kw["lower"].double()
    f = (low + (1 - low) * torch.sigmoid(proj[:, H * dim:2 * H * dim].double() + kw["f_bias"].double())).view(T, H, dim)
    return proj, kw, q, f, proj[:, 2 * H * dim:].double().view(T, H, vdim)


def hgrn2_direct(q, f, v, S):
    out = []
    for t in range(q.shape[0]):
        S = f[t][:, :, None] * S + (1 - f[t])[:, :, None] * v[t][:, None, :]
        out.append(torch.einsum("hkv,hk->hv", S, q[t]))
    return torch.stack(out), S


@pytest.mark.parametrize("dim", [8, 20, 32, 40, 64, 100, 128, 250])
@pytest.mark.parametrize("vdim", [24, 33, 64])
@pytest.mark.parametrize("dtype", [BF, F32])
def test_hgrn2_steps_and_portions_give_the_same_bits(ops, dim, vdim, dtype):
    """a sequence token by token in steps of its own (one kernel), beside a prompt portion (another) and in one call"""
    g, T, H = gen(dim + vdim), 19, 2
    proj, kw, q, f, v = hgrn2_inputs(g, T, H, dim, vdim, dtype)
    want, S = hgrn2_direct(q, f, v, torch.zeros(H, dim, vdim, device="cuda", dtype=torch.float64))
    i32 = lambda r: torch.tensor(r, dtype=torch.int32, device="cuda")
    whole = torch.full((4, H, dim, vdim), 9.0, device="cuda")
    ref = ops.hgrn2_scan(proj, whole, i32([(0, T, 0, 1)]), **kw)
    assert rel(ref.view(T, H, vdim), want) < 2e-6 and rel(whole[1], S) < 2e-6
    state, got = torch.full_like(whole, -3.0), []
    for t in range(T):
        if t % 3 == 2:      # beside three rows of another sequence
            got.append(ops.hgrn2_scan(torch.cat([proj[:3], proj[t:t + 1]]), state, i32([(0, 3, 0, 0), (3, 1, t, 2)]), **kw)[3:])
        else:               # alone or with another single row
            n = 1 + t % 2
            got.append(ops.hgrn2_scan(proj[t:t + 1].repeat(n, 1), state, i32([(0, 1, t, 2), (1, 1, 0, 3)][:n]), **kw)[:1])
    assert torch.equal(torch.cat(got), ref) and torch.equal(state[2], whole[1])


@pytest.mark.parametrize("seqs,H,dim,vdim,off", [(24, 16, 128, 64, 0), (24, 16, 64, 33, 0), (30, 40, 20, 30, 0), (2, 3, 128, 64, 1), (24, 16, 128, 64, 1),
                                                 (1, 2, 36, 34, 3)])
def test_wide_scans(ops, seqs, H, dim, vdim, off):
    """two and four columns per group of lanes (many sequences and heads), columns and channels that do not fill them, states
    that do not start on 16 bytes (off numbers past one)"""
    g, T = gen(dim + vdim), 18
    lens = [(5 * s) % T + 1 for s in range(seqs)]
    rows = [sum(lens[:s]) for s in range(seqs)]
    R, spans = sum(lens), torch.tensor([(rows[s], lens[s], 3 if s % 2 else 0, seqs - 1 - s) for s in range(seqs)], dtype=torch.int32, device="cuda")

    def state_of(*shape):
        flat = torch.randn(int(torch.tensor(shape).prod()) + off, generator=g, device="cuda")
        return flat[off:].view(*shape)

    proj, kw, q, f, v = hgrn2_inputs(g, R, H, dim, vdim)
    state = state_of(seqs, H, dim, vdim)
    start = state.double()
    got = ops.hgrn2_scan(proj, state, spans, **kw).view(R, H, vdim)
    x, B, Cm = randn(g, R, H, vdim), randn(g, R, 1, dim), randn(g, R, 1, dim)
    dt, z = randn(g, R, H), randn(g, R, H * vdim)
    A_log, bias, D = (torch.randn(H, generator=g, device="cuda") * 0.5 for _ in range(3))
    st2 = state_of(seqs, H, vdim, dim)
    start2 = st2.double()
    got2 = ops.ssd_scan(torch.cat([x.view(R, -1), B.view(R, -1), Cm.view(R, -1)], 1), dt, z, st2, spans, heads=H, vdim=vdim, nstate=dim, groups=1,
                        dt_bias=bias, A_log=A_log, D=D).view(R, H, vdim)
    step = torch.nn.functional.softplus(dt.double() + bias.double())
    gate = torch.nn.functional.silu(z.double()).view(R, H, vdim)
    for s in range(seqs):
        r, n, slot = rows[s], lens[s], seqs - 1 - s
        S = start[slot] if s % 2 else torch.zeros_like(start[slot])
        want, S = hgrn2_direct(q[r:r + n], f[r:r + n], v[r:r + n], S)
        assert rel(got[r:r + n], want) < 5e-6 and rel(state[slot], S) < 2e-6
        S = start2[slot] if s % 2 else torch.zeros_like(start2[slot])
        out = []
        for t in range(r, r + n):
            S = torch.exp(-torch.exp(A_log.double()) * step[t])[:, None, None] * S + (step[t][:, None] * x[t].double())[:, :, None] * B[t].double()
            out.append((S @ Cm[t, 0].double() + D.double()[:, None] * x[t].double()) * gate[t])
        assert rel(got2[r:r + n], torch.stack(out)) < 5e-6 and rel(st2[slot], S) < 2e-6


@pytest.mark.parametrize("dim", [20, 96, 126, 128])
def test_hgrn2_infinite_value(ops, dim):
    """channels past the head's do not turn an infinite value into NaN"""
    g, T, H, vdim = gen(dim), 6, 2, 24
    proj, kw, q, f, v = hgrn2_inputs(g, T, H, dim, vdim)
    proj[:, :H * dim] = proj[:, :H * dim].abs() + 0.5               # positive queries
    proj[2, 2 * H * dim + 7] = float("inf")
    for n in (T, 1):
        state, out = torch.zeros(1, H, dim, vdim, device="cuda"), []
        for t in range(0, T, n):
            out.append(ops.hgrn2_scan(proj[t:t + n], state, torch.tensor([(0, n, t, 0)], dtype=torch.int32, device="cuda"), **kw))
        out = torch.cat(out).view(T, H, vdim)
        assert torch.isinf(out[2:, 0, 7]).all() and torch.isfinite(out[:2]).all() and torch.isfinite(out[:, 0, :7]).all() and torch.isfinite(out[:, 1]).all()


# ---- ssd scans in chunks of 64 tokens ---------------------------------------------------------------------------
def ssd_inputs(lens, H, P, N, G, seed=3, gate=True, pad=8):
    """x | B | C behind a SiLU, step sizes and gates as a projection leaves them; odd slots start in mid-sequence"""
    g, T = gen(seed), sum(lens)
    wide = torch.randn(T, H * P + 2 * G * N + pad, generator=g, device="cuda")
    xbc = torch.nn.functional.silu(wide).to(BF)[:, :H * P + 2 * G * N]
    z = torch.randn(T, H * P, generator=g, device="cuda").to(BF) if gate else None
    dt = torch.randn(T, H + 1, generator=g, device="cuda").to(BF)[:, :H]
    kw = dict(heads=H, vdim=P, nstate=N, groups=G, dt_bias=torch.rand(H, generator=g, device="cuda") * 2.3 - 4.6,
              A_log=torch.log(1 + 15 * torch.rand(H, generator=g, device="cuda")), D=torch.randn(H, generator=g, device="cuda"))
    state = torch.randn(len(lens) + 1, H, P, N, generator=g, device="cuda")
    rows = [sum(lens[:s]) for s in range(len(lens))]
    seqs = torch.tensor([(rows[s], n, 7 if s % 2 else 0, len(lens) - s) for s, n in enumerate(lens)], dtype=torch.int32, device="cuda")
    return xbc, dt, z, state, seqs, kw


def ssd_float64(xbc, dt, z, state, seqs, kw):
    H, P, N, G = kw["heads"], kw["vdim"], kw["nstate"], kw["groups"]
    u, S_all = xbc.double(), state.double()
    out = torch.empty(u.shape[0], H, P, dtype=torch.float64, device="cuda")
    step = torch.nn.functional.softplus(dt.double() + kw["dt_bias"].double())
    A = torch.exp(kw["A_log"].double())
    for r, n, pos, slot in seqs.tolist():
        S = S_all[slot] if pos else torch.zeros_like(S_all[slot])
        for t in range(r, r + n):
            x = u[t, :H * P].view(H, P)
            B, Cm = (u[t, H * P + i * G * N:H * P + (i + 1) * G * N].view(G, N).repeat_interleave(H // G, 0) for i in range(2))
            S = torch.exp(-A * step[t])[:, None, None] * S + (step[t][:, None] * x)[:, :, None] * B[:, None]
            out[t] = torch.einsum("hpn,hn->hp", S, Cm) + kw["D"].double()[:, None] * x
        S_all[slot] = S
    out = out.view(u.shape[0], -1)
    return (out if z is None else out * torch.nn.functional.silu(z.double())), S_all


@pytest.mark.parametrize("lens,H,P,N,G,gate", [([48], 2, 64, 128, 1, True), ([63, 64, 65], 4, 32, 128, 2, True), ([129, 47, 1, 192], 2, 48, 128, 2, False),
                                               ([200], 3, 16, 128, 1, True), ([70, 48], 2, 96, 64, 1, True), ([66], 150, 32, 128, 5, True)])
def test_ssd_chunks(ops, lens, H, P, N, G, gate):
    """portions at the chunks' edges, beside shorter ones that go token by token; 16 and 32 columns per CTA"""
    xbc, dt, z, state, seqs, kw = ssd_inputs(lens, H, P, N, G, gate=gate)
    want, S = ssd_float64(xbc, dt, z, state, seqs, kw)
    got_state = state.clone()
    got = ops.ssd_scan(xbc, dt, z, got_state, seqs, **kw)
    # fp32 roundings of a sum of decaying terms: a few units of 6e-8
    assert rel(got, want) < 5e-7 and rel(got_state, S) < 5e-7 and torch.equal(got_state[0], state[0])
    assert rel(ops.ssd_scan(xbc, dt, z, state.clone(), seqs, out_dtype=BF, **kw), want) < 4e-3
    # a sequence's numbers depend neither on the batch nor on the others' lengths
    for s, (r, n, pos, slot) in enumerate(seqs.tolist()):
        one = state.clone()
        alone = ops.ssd_scan(xbc[r:r + n], dt[r:r + n], None if z is None else z[r:r + n], one, torch.tensor([(0, n, pos, slot)], dtype=torch.int32, device="cuda"), **kw)
        assert torch.equal(alone, got[r:r + n]) and torch.equal(one[slot], got_state[slot])


@pytest.mark.parametrize("odd", [False, True])
def test_ssd_chunks_same_bits_in_either_width(ops, odd):
    """one sequence of 32 heads x 64 takes CTAs of 16 columns, three take CTAs of 32: the same bits, also beside an infinite
    value, whose 16 columns alone are walked token by token"""
    H, P, N = 32, 64, 128
    xbc, dt, z, state, seqs, kw = ssd_inputs([200, 150, 100], H, P, N, 1)
    if odd:
        xbc[70, 3 * P + 18] = float("inf")
        state[2, 5, 40, 7] = float("nan")                             # of the second sequence, which starts in mid-sequence
    batch = state.clone()
    got = ops.ssd_scan(xbc, dt, z, batch, seqs, **kw)
    assert torch.isfinite(got).all() != odd
    for r, n, pos, slot in seqs.tolist():
        one = state.clone()
        alone = ops.ssd_scan(xbc[r:r + n], dt[r:r + n], z[r:r + n], one, torch.tensor([(0, n, pos, slot)], dtype=torch.int32, device="cuda"), **kw)
        for a, b in ((alone, got[r:r + n]), (one[slot], batch[slot])):
            assert torch.equal(torch.nan_to_num(a, 1.5, 2.5, 3.5), torch.nan_to_num(b, 1.5, 2.5, 3.5))


def test_ssd_chunks_after_any_decay(ops):
    """steps that forget the state at once and steps that keep it, in one chunk"""
    xbc, dt, z, state, seqs, kw = ssd_inputs([100, 100], 2, 32, 128, 1)
    dt = dt.float() * 1.0
    dt[10::7], dt[13::11] = 60.0, -40.0
    dt = dt.to(BF)
    want, S = ssd_float64(xbc, dt, z, state, seqs, kw)
    got = ops.ssd_scan(xbc, dt, z, state, seqs, **kw)
    assert rel(got, want) < 5e-7 and rel(state[1:], S[1:]) < 5e-7


@pytest.mark.parametrize("rows,copies", [(60, 2), (100, 5), (48, 40)])
def test_ssd_chunks_of_sequences_that_share_their_rows(ops, rows, copies):
    """several states advanced over the same rows: more long sequences than rows of their own would allow"""
    H, P, N = 2, 32, 128
    xbc, dt, z, state, _, kw = ssd_inputs([rows], H, P, N, 1)
    state = torch.randn(1, H, P, N, device="cuda", generator=gen(2)).repeat(copies + 1, 1, 1, 1)
    seqs = torch.tensor([(0, rows, 5, copies - s) for s in range(copies)], dtype=torch.int32, device="cuda")
    want, S = ssd_float64(xbc, dt, z, state, seqs[:1], kw)
    untouched = state[0].clone()
    got = ops.ssd_scan(xbc, dt, z, state, seqs, **kw)
    assert rel(got, want) < 5e-7 and torch.equal(state[0], untouched)
    for slot in range(1, copies + 1):
        assert rel(state[slot], S[copies]) < 5e-7


@pytest.mark.parametrize("where", ["x", "B", "C", "dt", "z", "state", "nan"])
def test_ssd_chunks_infinite_numbers(ops, where):
    """rows before an infinite number stay as they are, the others are what the recurrence makes of it"""
    H, P, N = 2, 32, 128
    xbc, dt, z, state, seqs, kw = ssd_inputs([150, 70], H, P, N, 1)
    inf, r = float("inf"), 80
    if where == "x": xbc[r, 5] = inf
    if where == "nan": xbc[r, 5] = float("nan")
    if where == "B": xbc[r, H * P + 9] = -inf
    if where == "C": xbc[r, H * P + N + 9] = inf
    if where == "dt": dt[r, 1] = inf
    if where == "z": z[r, 3], z[r + 1, 3] = inf, -inf
    if where == "state": state[1, 0, 3, 4] = inf
    from vila_b200 import _lib
    lib, rows = _lib.load(), []
    call = lib.vila_ssd_scan_rows
    try:
        for token_by_token in (False, True):
            if token_by_token:
                lib.vila_ssd_scan_rows = lambda p, n, stream: lib.vila_ssd_scan(p, stream)
            st = state.clone()
            rows.append((ops.ssd_scan(xbc, dt, z, st, seqs, **kw), st))
    finally:
        lib.vila_ssd_scan_rows = call
    assert not torch.isfinite(rows[1][0]).all()
    for a, b in zip(*rows):
        ok = torch.isfinite(b)
        assert torch.equal(torch.isnan(a), torch.isnan(b)) and torch.equal(torch.isfinite(a), ok) and rel(a[ok], b[ok].double()) < 5e-7


@pytest.mark.parametrize("M,N,K", [(1, 128, 2048), (8, 130, 2056), (9, 129, 4096), (16, 4097, 4104), (16, 200, 8192), (3, 17000, 1032), (5, 33000, 512), (16, 333, 264),
                                   (2, 144, 8), (3, 1024, 1024), (8, 7104, 256), (4, 7120, 1024), (9, 4096, 256), (7, 4112, 248), (16, 2048, 128)])
def test_few_rows_stream(ops, M, N, K):
    """CTAs that stay and those that don't: ragged columns, a last tile of one weight row, token rows that do not fit in shared memory"""
    g = gen(M + N + K)
    a, w, b = randn(g, M, K + 8)[:, :K], randn(g, N, K), randn(g, N)
    ref = a.double() @ w.double().T
    got = ops.glinear(a, w, out_dtype=F32)
    # about 32 roundings of at most 2^-24 each, taken as independent
    assert rel(got, ref) < 32 ** 0.5 * 2.0 ** -24
    assert rel(ops.glinear(a, w, bias=b, act=ops.ACT_RELU2, out_dtype=F32), torch.relu(ref + b.double()) ** 2) < 3 * 32 ** 0.5 * 2.0 ** -24
    # a row's sums do not depend on the other rows
    assert torch.equal(ops.glinear(a[:1], w, out_dtype=F32), got[:1])
    # products of one sign: truncations of 16 terms at 2^-24 of their sum (a bias), the additions after them rounded at no more
    # than 2^-24 of the whole in each of four levels, and the last bit
    pos = ops.glinear(a.abs(), w.abs(), out_dtype=F32)
    want = a.double().abs() @ w.double().abs().T
    assert rel(pos, want) < (1 + 5 ** 0.5) * 2.0 ** -24 and float(((pos.double() - want) / want).mean().abs()) < 2.0 ** -24
    if N % 2 == 0:
        z = ref / K ** 0.5
        want = torch.nn.functional.silu(z[:, 0::2]) * z[:, 1::2]
        assert rel(ops.glinear((a.float() / K ** 0.5).to(BF), w, swiglu=True, out_dtype=F32), want) < 2.0 ** -7   # a is rounded once more


@pytest.mark.parametrize("T,E,top,N,K,shared", [(16, 40, 4, 256, 1024, True), (16, 3, 2, 1000, 2048, True), (12, 70, 5, 130, 4096, False), (21, 33, 3, 144, 1040, False),
                                                (1, 9, 4, 1040, 1024, True), (16, 4, 4, 200, 704, True)])
def test_few_pairs_stream(ops, T, E, top, N, K, shared):
    """groups without rows and with more than a pass of eight, rows that several pairs share or do not"""
    g = gen(T + E + N)
    idx = torch.rand(T, E, generator=g, device="cuda").topk(min(top, E)).indices.to(torch.int32)
    top = idx.shape[1]
    idx[:, 0] = 1                                                     # group 1 has T pairs, group 0 none but by chance
    seg, srt = ops.moe_group(idx, E)
    w = randn(g, E, N, K)
    a = randn(g, T if shared else T * top, K)
    wt, scale = torch.rand(T * top, generator=g, device="cuda"), torch.rand(a.shape[0], generator=g, device="cuda")
    rows = a.double().repeat_interleave(top, 0) if shared else a.double()
    ref = torch.einsum("rk,rnk->rn", rows, w[idx.view(-1).long()].double())
    kw = dict(groups=E, seg=seg, a_rows=srt, a_row_div=top if shared else 1, out_dtype=F32)
    got = ops.glinear(a, w, o_rows=srt, row_scale=wt, out_rows_total=T * top, **kw)
    assert rel(got, ref * wt.double()[:, None]) < 2 * 32 ** 0.5 * 2.0 ** -24
    glu = ops.glinear(a, w, glu_clamp=(1.702, 7.0), **kw)              # sorted order
    z = ref[srt.long()]
    gt, u = torch.clamp_max(z[:, 0::2], 7.0), torch.clamp(z[:, 1::2], -7.0, 7.0)
    assert rel(glu, gt * torch.sigmoid(1.702 * gt) * (u + 1)) < 1e-6


@pytest.mark.parametrize("T,width,identity", [(1, 2048, "some"), (8, 2048, "some"), (16, 2048, "some"), (16, 1024, "some"), (16, 2048, "all"), (8, 1024, "all")])
def test_few_pairs_without_a_group(ops, T, width, identity):
    """choices of identity outputs are in no segment: 28 experts + 4 such outputs, the sorted list ends before its storage does.
    The positions behind it name another pair here, whose weight is infinite and whose row is NaN: nothing of them may count."""
    E, top, ff = 28, 4, 1024
    g = gen(T + width)
    idx = torch.rand(T, E + 4, generator=g, device="cuda").topk(top).indices.to(torch.int32)
    idx[:, -1] = E + 1                                                # a pair without a group in every row
    if identity == "all":
        idx[:] = E
    seg, srt = ops.moe_group(idx, E)
    live = int((idx < E).sum())
    assert int(seg[-1]) == live < T * top
    srt[live:] = top - 1                                              # pair of row 0 that is in no segment
    up, down, h = randn(g, E, ff, width), randn(g, E, width, ff) * 0.05, randn(g, T, width)
    wt = torch.rand(T * top, generator=g, device="cuda")
    wt[top - 1] = float("inf")
    pairs, expert = srt[:live].long(), idx.view(-1)[srt[:live].long()].long()
    act = ops.glinear(h, up, groups=E, seg=seg, a_rows=srt, a_row_div=top, act=ops.ACT_GELU_ERF)
    want = torch.nn.functional.gelu(torch.einsum("rk,rnk->rn", h.double()[pairs // top], up[expert].double()))
    if live:
        assert rel(act[:live], want) < 2.0 ** -8
    act[live:] = float("nan")
    rows = torch.zeros(T * top, width, device="cuda")
    ops.glinear(act, down, groups=E, seg=seg, o_rows=srt, row_scale=wt, out=rows)
    want = torch.zeros(T * top, width, dtype=torch.float64, device="cuda")
    want[pairs] = torch.einsum("rk,rnk->rn", act[:live].double(), down[expert].double()) * wt.double()[pairs, None]
    assert torch.equal(rows[want.abs().sum(1) == 0], torch.zeros_like(rows[want.abs().sum(1) == 0]))
    if live:
        assert rel(rows, want) < 2 * 32 ** 0.5 * 2.0 ** -24
