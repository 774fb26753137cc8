"""Kernels at the sizes where a new tile, copy width or split can go wrong, against plain float64 references."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def ops():
    from vllm_lite_b200.csrc import ops as o
    return o


# every tile of the float32 product (8 x 32, 32 x 32, 64 x 64, 128 x 128), its edges, K with and without 16-byte copies
@pytest.mark.parametrize("N,K", [(1, 1), (31, 4), (33, 63), (320, 96), (333, 97), (700, 260), (8193, 68)])
@pytest.mark.parametrize("M", [1, 8, 9, 16, 17, 33, 64, 65, 130])
def test_gemm_f32_tiles(M, N, K):
    gen = torch.Generator(device=DEV).manual_seed(M * 131 + N + K)
    a, w = torch.randn(M, K, device=DEV, generator=gen), torch.randn(N, K, device=DEV, generator=gen)
    out = torch.full((M, N), float("nan"), device=DEV)
    ops().gemm_f32(a, w, out)
    ref = a.double() @ w.double().T
    # K roundings of a running sum of products of the same sizes: at most K 2^-24 sum |a| |w|
    bound = (K + 1) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T)
    assert bool(((out.double() - ref).abs() <= bound).all())
    one = torch.empty(1, N, device=DEV)
    ops().gemm_f32(a[M - 1:].contiguous(), w, one)
    assert torch.equal(one[0], out[M - 1])               # whichever tile made the row


# the activation in the product's epilogue: the bits of the product and the activation by themselves, in every tile
@pytest.mark.parametrize("I,K,group", [(1, 1, 0), (7, 63, 0), (160, 96, 8), (161, 97, 0), (24, 64, 4), (352, 260, 16), (4104, 68, 8)])
@pytest.mark.parametrize("M", [1, 8, 9, 16, 17, 64, 65, 130])
def test_gemm_f32_with_its_activation(M, I, K, group):
    gen = torch.Generator(device=DEV).manual_seed(M * 131 + I + K)
    a, w = torch.randn(M, K, device=DEV, generator=gen), torch.randn(2 * I, K, device=DEV, generator=gen)
    product, want = torch.empty(M, 2 * I, device=DEV), torch.empty(M, I, device=DEV)
    out = torch.full((M, I), float("nan"), device=DEV)
    ops().silu_mul(ops().gemm_f32(a, w, product), want, group)
    ops().gemm_f32(a, w, out, swiglu=True, group=group)
    assert torch.equal(out, want)


# tiles of 16, 32 and 48 rows of W, one to three of 16 rows of A, their edges, warps without a block of K and K's last block cut
@pytest.mark.parametrize("N,K", [(1, 8), (24, 72), (64, 2048), (2368, 520), (2370, 136), (4752, 1032), (7104, 64)])
@pytest.mark.parametrize("M", [1, 9, 16, 17, 32, 33, 48])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_product_of_few_rows(M, N, K, out_dtype):
    gen = torch.Generator(device=DEV).manual_seed(M * 131 + N + K)
    a = torch.randn(M, K, device=DEV, generator=gen).bfloat16()
    w = (torch.randn(N, K, device=DEV, generator=gen) / K ** 0.5).bfloat16()
    err = torch.zeros(1, dtype=torch.int32, device=DEV)
    out = torch.full((M + 1, N), 7.0, device=DEV, dtype=out_dtype)
    ops().gemm_bf16_few(a, w, out[:M], err)
    ref, size = a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
    # float32 sums of K exact products, then one rounding to the result's type
    bound = (K + 8) * 2.0 ** -24 * size + (2.0 ** -8 * ref.abs() if out_dtype == torch.bfloat16 else 0)
    assert bool(((out[:M].double() - ref).abs() <= bound).all()) and bool((out[M:] == 7.0).all()) and not int(err)
    if N % 16 == 0:
        act = torch.empty(M, N // 2, device=DEV, dtype=out_dtype)
        ops().gemm_bf16_few(a, w, act, err, swiglu=True)
        g, u = (ref.view(M, -1, 2, 8)[:, :, i].reshape(M, -1) for i in (0, 1))
        og, ou = ((K + 8) * 2.0 ** -24 * size.view(M, -1, 2, 8)[:, :, i].reshape(M, -1) for i in (0, 1))
        ref = g / (1 + torch.exp(-g)) * u
        # |silu'| < 1.1, |silu(g)| <= |g|, and a float32 exponential, quotient and product
        bound = 1.2 * og * u.abs() + g.abs() * ou + 2.0 ** -20 * ref.abs() + (2.0 ** -8 * ref.abs() if out_dtype == torch.bfloat16 else 0) + 1e-30
        assert bool(((act.double() - ref).abs() <= bound).all())


# a block a row and a warp a row (4,000 and more), columns beyond a round of accesses, sums over one to five choices: the arithmetic in order
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("T,K,top,scale", [(5, 96, 2, True), (1999, 264, 2, True), (1400, 2056, 3, False), (900, 4104, 5, True), (1400, 100, 3, True)])
def test_sorted_rows_and_their_sums(T, K, top, scale, dtype):
    E, bm = 8, 16
    gen = torch.Generator(device=DEV).manual_seed(T + K)
    ids = torch.rand(T, E, device=DEV, generator=gen).topk(top).indices.to(torch.int32).contiguous()
    weights, h = torch.rand(T, top, device=DEV, generator=gen), torch.randn(T, K, device=DEV, generator=gen).to(dtype)
    cap = ops().moe_sorted_rows(T * top, E, bm)
    order, place = (torch.empty(n, dtype=torch.int32, device=DEV) for n in (cap, T * top))
    ops().moe_align(ids, E, bm, order, torch.empty(cap // bm, dtype=torch.int32, device=DEV), place)
    rows = ops().moe_gather(h, order, weights, top, torch.full((cap, K), 7.0, device=DEV, dtype=dtype), scale)
    pair = order.long().clamp(min=0)
    want = h[pair // top].float() * (weights.view(-1)[pair][:, None] if scale else 1.0)
    assert torch.equal(rows, torch.where(order[:, None] >= 0, want, 0.0).to(dtype))
    out = ops().moe_combine(rows, place, weights, top, torch.empty(T, K, device=DEV, dtype=dtype), True)
    ref = (rows[place.long()].double().view(T, top, K) * weights.double()[:, :, None])
    # float32 products and sums, then one rounding to the result's type
    bound = 2 * top * 2.0 ** -24 * ref.abs().sum(1) + (2.0 ** -8 if dtype == torch.bfloat16 else 0) * ref.sum(1).abs() * 1.01 + 1e-30
    assert bool(((out.double() - ref.sum(1)).abs() <= bound).all())


@pytest.mark.parametrize("M,N,K", [(129, 256, 128), (128, 640, 2048), (300, 384, 136)])      # few tiles: 128 columns wide
def test_tcgen05_product_with_few_tiles(M, N, K):
    gen = torch.Generator(device=DEV).manual_seed(M + N + K)
    a = torch.randn(M, K, device=DEV, generator=gen).bfloat16()
    w = (torch.randn(N, K, device=DEV, generator=gen) / K ** 0.5).bfloat16()
    err, out = torch.zeros(1, dtype=torch.int32, device=DEV), torch.full((M, N), float("nan"), device=DEV)
    ops().gemm_bf16_tc5(a, w, out, err)
    bound = (K + 8) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T)
    assert bool(((out.double() - a.double() @ w.double().T).abs() <= bound).all()) and not int(err)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("T,I,group", [(1, 8, 0), (3, 4096, 0), (5, 12, 0), (2, 7, 0), (3, 64, 8), (3, 64, 16), (5, 36, 4), (7, 48, 24)])
def test_silu_mul_layouts(T, I, group, dtype):
    gu = (torch.randn(T, 2 * I, device=DEV) * 4).to(dtype)
    out = torch.empty(T, I, device=DEV, dtype=dtype)
    ops().silu_mul(gu, out, group=group)
    parts = gu.double().view(T, -1, 2, group or I)
    g, u = parts[:, :, 0].reshape(T, I), parts[:, :, 1].reshape(T, I)
    ref = g / (1 + torch.exp(-g)) * u
    rel = 2.0 ** -8 if dtype == torch.bfloat16 else 1e-6      # one rounding / a handful of them
    assert bool(((out.double() - ref).abs() <= rel * ref.abs() + 1e-30).all())


# few outputs are made one by one, many by eights where the layout allows it: 196,608 outputs in bfloat16 and 327,680 in float32 on, those
# without an exponential always
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("T,I,group", [(3, 64, 0), (3, 64, 8), (5, 36, 4), (409, 480, 24), (410, 480, 24), (410, 792, 0), (415, 792, 8), (300, 1100, 0)])
@pytest.mark.parametrize("act", ["silu", "relu", "capped"])
def test_gated_activations_by_ones_and_by_eights(T, I, group, act, dtype):
    o, alpha = ops(), float(torch.tensor(1.7)) if act == "capped" else 1.0       # 1.7 as the kernel gets it, in float32
    gu, out = (torch.randn(T, 2 * I, device=DEV) * 4).to(dtype), torch.empty(T, I, device=DEV, dtype=dtype)
    bias = torch.randn(2 * I, device=DEV) if act == "capped" else None
    o._check(o._fn("activation", "vl_gated_act")(gu.data_ptr(), out.data_ptr(), o.dtype_code(dtype), T, I, group, ("silu", "relu", "capped").index(act),
                                                 alpha, 5.0, 1.0, bias.data_ptr() if act == "capped" else None, o._stream()), "vl_gated_act")
    parts = (gu.float() + bias if act == "capped" else gu).double().view(T, -1, 2, group or I)
    g, u = parts[:, :, 0].reshape(T, I), parts[:, :, 1].reshape(T, I)
    if act == "capped":
        g, u = g.clamp(max=5), u.clamp(-5, 5) + 1
    ref = g.clamp(min=0) * u if act == "relu" else g / (1 + torch.exp(-alpha * g)) * u
    # the exponential's argument is rounded, an error of alpha |g| 2^-24 in its result; a handful of roundings more (at most 8 x 2^-24: the
    # exponential 2^-22, the sum, the quotient, u + 1, the product), and the output's own (eight bits: at most 2^-8 of the number)
    rel = (alpha * float(g.abs().max()) + 8) * 2.0 ** -24 + (2.0 ** -8 if dtype == torch.bfloat16 else 0)
    assert bool(((out.double() - ref).abs() <= rel * ref.abs() + 1e-30).all())


# the persistent decode attention: runs of key tiles that cut items anywhere, places without keys, a long item beside short
# ones (few pieces allowed: runs as long as that item asks), one page and several a tile, a window, sinks
@pytest.mark.parametrize("lengths,bound,pieces", [
    ([1], 64, 2), ([64, 65, 63], 128, 2), ([0, 200, 0, 1, 130], 256, 3), ([4000] + [3] * 9, 4096, 2), ([4000] + [3] * 9, 4096, 6),
    ([(37 * i * i) % 700 for i in range(70)], 2048, 6), ([300, 900, 64, 128, 1, 2047], 2048, 6), ([900, 2500, 17], 1024, 4),
    ([(13 * i) % 160 for i in range(500)], 256, 3)])     # more places than a block's threads count in one go
@pytest.mark.parametrize("hd,page,window,sink", [(128, 64, None, False), (64, 16, 150, False), (128, 128, 65, True), (64, 64, None, True)])
def test_streaming_decode_attention(lengths, bound, pieces, hd, page, window, sink):
    nq, nkv, T, scale = 8, 2, len(lengths), hd ** -0.5
    gen = torch.Generator(device=DEV).manual_seed(sum(lengths) + hd)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=gen).to(torch.bfloat16)
    blocks = -(-max(max(lengths), bound) // page)
    table = torch.randperm(T * blocks, device=DEV, generator=gen).to(torch.int32).view(T, blocks)
    kc, vc = rnd(T * blocks, nkv, page, hd), rnd(T * blocks, nkv, page, hd)
    qkv = rnd(T, (nq + 2 * nkv) * hd)
    sinks = torch.randn(nq, device=DEV, generator=gen) if sink else None
    pos = torch.tensor([n - 1 for n in lengths], dtype=torch.int32, device=DEV)
    req = torch.arange(T, dtype=torch.int32, device=DEV)
    err = torch.zeros(1, dtype=torch.int32, device=DEV)
    acc, ml = torch.full((T * nq * pieces * hd,), float("nan"), device=DEV), torch.full((T * nq * pieces * 2,), float("nan"), device=DEV)
    arrivals = torch.zeros(ops().flash_decode_arrivals(T, nq, nkv), dtype=torch.int32, device=DEV)
    out = rnd(T, nq * hd)
    for _ in range(2):                                   # twice on the same counters
        ops().flash_decode(qkv, out, kc, vc, table, req, pos, nq, nkv, hd, scale, window, bound, acc, ml, err, chunk=-(-bound // pieces // 64) * 64,
                           stream_kernel=True, arrivals=arrivals, sinks=sinks)
    limit = -(-bound // (-(-bound // pieces // 64) * 64)) * (-(-bound // pieces // 64) * 64)
    assert int(arrivals.abs().sum()) == 0
    assert bool(int(err) & 0x10) == any(n > limit for n in lengths) and not int(err) & ~0x10
    for t, n in enumerate(lengths):
        got = out[t].double().view(nq, hd)
        if n == 0 or n > limit:
            assert not got.any()
            continue
        lo = max(0, n - window) if window else 0
        rows = lambda c: c[table[t].long()].double().transpose(0, 1).reshape(nkv, -1, hd)[:, lo:n].repeat_interleave(nq // nkv, 0)
        s = torch.einsum("hd,hnd->hn", qkv[t, :nq * hd].double().view(nq, hd), rows(kc)) * scale
        if sinks is not None:
            s = torch.cat([s, sinks.double()[:, None]], 1)
        p = torch.softmax(s, -1)[:, :n - lo]
        ref, size = torch.einsum("hn,hnd->hd", p, rows(vc)), torch.einsum("hn,hnd->hd", p, rows(vc).abs())
        # probabilities and the result are rounded to bfloat16, the exponentials are good to about 2^-22
        assert bool(((got - ref).abs() <= 2.0 ** -8 * ref.abs() + 2.0 ** -8 * size + 1e-6).all()), (t, n)


# rows of the output, scratch and numbers of pieces that begin anywhere, among them a place without keys and one beyond the bound
@pytest.mark.parametrize("off", [1, 3, 8])
def test_streaming_decode_attention_off_the_boundaries(off):
    nq, nkv, hd, page, lengths, bound, pieces = 8, 2, 128, 64, [300, 0, 1000, 17, 2000], 1024, 6
    T, gen = len(lengths), torch.Generator(device=DEV).manual_seed(off)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=gen).to(torch.bfloat16)
    blocks = 2048 // page
    table = torch.randperm(T * blocks, device=DEV, generator=gen).to(torch.int32).view(T, blocks)
    kc, vc, qkv = rnd(T * blocks, nkv, page, hd), rnd(T * blocks, nkv, page, hd), rnd(T, (nq + 2 * nkv) * hd)
    pos, req = torch.tensor([n - 1 for n in lengths], dtype=torch.int32, device=DEV), torch.arange(T, dtype=torch.int32, device=DEV)
    arrivals = torch.zeros(ops().flash_decode_arrivals(T, nq, nkv), dtype=torch.int32, device=DEV)

    def run(at):
        err, n = torch.zeros(1, dtype=torch.int32, device=DEV), T * nq * pieces
        whole = torch.full((T * nq * hd + 16,), 7.0, device=DEV, dtype=torch.bfloat16)
        out = whole[at:at + T * nq * hd].view(T, nq * hd)
        acc, ml = torch.empty(n * hd + at, device=DEV)[at:], torch.empty(n * 2 + at, device=DEV)[at:]
        ops().flash_decode(qkv, out, kc, vc, table, req, pos, nq, nkv, hd, hd ** -0.5, None, bound, acc, ml, err, chunk=bound,
                           stream_kernel=True, arrivals=arrivals)
        assert int(err) == 0x10 and bool((whole[:at] == 7).all()) and bool((whole[at + T * nq * hd:] == 7).all())
        return out

    assert torch.equal(run(off), run(0))


# the same with dependent launches on: positions that a kernel ahead writes (itself behind a long one) are waited for, those that a copy
# brought may be read early (`settled`); kernels that write the cache stand ahead in both
@pytest.mark.parametrize("made_by", ["kernel", "copy"])
def test_streaming_decode_attention_behind_dependent_launches(made_by):
    nq, nkv, hd, page, T, bound, pieces = 8, 2, 128, 64, 24, 512, 6
    gen = torch.Generator(device=DEV).manual_seed(3)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=gen)
    blocks = bound // page
    table = torch.randperm(T * blocks, device=DEV, generator=gen).to(torch.int32).view(T, blocks)
    caches = [[rnd(T * blocks, nkv, page, hd).to(torch.bfloat16) for _ in range(2)] for _ in range(3)]
    qkv, inv = rnd(T, (nq + 2 * nkv) * hd).to(torch.bfloat16), torch.rand(hd // 2, device=DEV, generator=gen)
    order = torch.randperm(T, generator=torch.Generator().manual_seed(4)).to(torch.int32)
    where = 16 * order                                   # what sorting one row an expert by expert gives, tiles of 16 rows
    slots = torch.tensor([int(table[t, int(p) // page]) * page + int(p) % page for t, p in enumerate(where)], dtype=torch.int32, device=DEV)
    req, ids, pinned = torch.arange(T, dtype=torch.int32, device=DEV), order.to(DEV).view(T, 1), where.pin_memory()
    err = torch.zeros(1, dtype=torch.int32, device=DEV)
    acc, ml = torch.empty(T * nq * pieces * hd, device=DEV), torch.empty(T * nq * pieces * 2, device=DEV)
    arrivals = torch.zeros(ops().flash_decode_arrivals(T, nq, nkv), dtype=torch.int32, device=DEV)
    cap = ops().moe_sorted_rows(T, T, 16)
    rows, tiles = torch.empty(cap, dtype=torch.int32, device=DEV), torch.empty(cap // 16, dtype=torch.int32, device=DEV)
    big, product = rnd(2048, 4096), torch.empty(2048, 2048, device=DEV)

    def run(pdl):
        pos = torch.zeros(T, dtype=torch.int32, device=DEV)
        heads, outs = qkv.clone(), [torch.empty(T, nq * hd, device=DEV, dtype=torch.bfloat16) for _ in caches]
        torch.cuda.synchronize()
        ops().set_pdl(pdl)
        try:
            copied = pinned.to(DEV, non_blocking=True)
            if made_by == "copy":
                pos = copied
            ops().gemm_f32(big, big[:2048], product)     # hundreds of microseconds
            if made_by == "kernel":
                ops().moe_align(ids, T, 16, rows, tiles, pos)
            for (k, v), out in zip(caches, outs):
                ops().qk_norm_rope_write(heads, copied, slots, None, None, 0.0, inv, hd, k, v, nq, nkv, hd, err)
                ops().flash_decode(heads, out, k, v, table, req, pos, nq, nkv, hd, hd ** -0.5, None, bound, acc, ml, err, chunk=bound,
                                   stream_kernel=True, arrivals=arrivals, settled=made_by == "copy")
        finally:
            ops().set_pdl(False)
        assert torch.equal(pos.cpu(), where) and int(err) == 0 and not arrivals.any()
        return outs

    plain = run(False)
    for _ in range(5):
        assert all(torch.equal(a, b) for a, b in zip(run(True), plain))


def decayed_memory(r, k, v, w, u, S):
    """float64, one request: r, k, w [T, H, D], v [T, H, P], u [H, D], S [H, D, P]; (outputs [T, H, P], the state behind them)."""
    out = torch.empty(v.shape, dtype=torch.float64, device=DEV)
    for t in range(r.shape[0]):
        kv = k[t][:, :, None] * v[t][:, None]
        out[t] = torch.einsum("hdp,hd->hp", S + u[:, :, None] * kv, r[t])
        S = w[t][:, :, None] * S + kv
    return out, S


# portions on both sides of 96 tokens and of whole chunks, heads of one tile and two, decays from nothing kept to all kept, a state carried over
@pytest.mark.parametrize("H,D,P", [(1, 4, 4), (2, 12, 20), (2, 64, 64), (3, 64, 36), (2, 128, 128), (1, 100, 68)])
@pytest.mark.parametrize("lengths", [[96], [95, 128, 97], [129, 1, 200], [7, 191]])
@pytest.mark.parametrize("decays", ["mixed", "strong", "zeros"])
def test_decay_chunks(H, D, P, lengths, decays):
    gen = torch.Generator(device=DEV).manual_seed(D * 7 + sum(lengths))
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=gen)
    T, B, eps = sum(lengths), len(lengths), 1e-5
    cu = torch.tensor([sum(lengths[:i]) for i in range(B + 1)], dtype=torch.int32, device=DEV)
    slots = torch.arange(B, 0, -1, dtype=torch.int32, device=DEV)
    u, norm = rnd(H * D) * 0.5, 1 + 0.1 * rnd(H * P)
    state = torch.zeros(B + 1, ops().decay_state_floats(H, D, P) + 4, device=DEV)
    S = [torch.zeros(H, D, P, dtype=torch.float64, device=DEV) for _ in lengths]
    for turn in range(2):                                # the second portions start from what the first ones left
        r, k, v, gate = rnd(T, H * D + 4), rnd(T, H * D), rnd(T, H * P), rnd(T, H * P + 8).to(torch.bfloat16)
        w = {"mixed": torch.exp(-torch.exp(2 * rnd(T, H * D) - 2)), "strong": torch.exp(-torch.exp(rnd(T, H * D) + 2)),
             "zeros": (rnd(T, H * D) > 0).float()}[decays]
        out = torch.full((T, H * P), float("nan"), device=DEV, dtype=torch.bfloat16)
        o = torch.empty(T, H * P, device=DEV)
        scan = (r, 4), (k, 0), (v, 0), (w, 0), u, state, 4, cu, slots
        walked = state.clone()
        ops().decay_scan(*scan[:5], walked, *scan[6:], o, H, D, P)       # the walk over everything, beside it
        if min(lengths) < ops().DECAY_MIN_CHUNK:
            o2 = torch.empty(T, H * P, device=DEV)
            ops().decay_scan(*scan, o2, H, D, P, longest=ops().DECAY_MIN_CHUNK - 1)
        chunks = ops().decay_chunks_of(lengths)
        scratch = torch.full((ops().decay_chunk_floats(chunks, H, D, P),), float("nan"), device=DEV)
        ops().decay_chunks(*scan, chunks, scratch, gate, 8, norm, eps, out, H, D, P)
        for b, n in enumerate(lengths):
            at = slice(int(cu[b]), int(cu[b]) + n)
            heads = lambda x, m: x[at].double().view(n, H, m)
            want, S[b] = decayed_memory(heads(r[:, 4:].contiguous(), D), heads(k, D), heads(v, P), heads(w, D), u.double().view(H, D), S[b])
            if n < ops().DECAY_MIN_CHUNK:
                assert torch.equal(o2[at], o[at]) and out[at].isnan().all()
                continue
            y = want / torch.sqrt((want * want).mean(-1, keepdim=True) + eps) * norm.double().view(H, P)
            y = y * torch.nn.functional.silu(heads(gate[:, 8:].contiguous(), P))
            assert float((heads(out, P) - y).norm() / y.norm()) <= 2.0 ** -8      # the result's rounding
        # float32 inside: the states as near to 64 bits as the walk's, up to a small factor
        native = lambda st, b: st[int(slots[b]), 4:]
        for b in range(B):
            err = [float((state_of(native(st, b), H, D, P) - S[b]).norm() / S[b].norm()) for st in (state, walked)]
            assert err[0] <= 2 * err[1] + 3e-7, (b, err)
            assert torch.equal(state[:, :4], walked[:, :4])


# a token's numbers reach its own and later outputs only, finite or not: every place in a group of four tokens, both halves of a chunk, the
# next chunk; heads whose states have rows for all of a block's threads and heads that have not
@pytest.mark.parametrize("D,P", [(4, 4), (20, 36), (64, 64), (128, 128)])
@pytest.mark.parametrize("which", ["k", "v", "w"])
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_decay_chunks_are_causal_for_numbers_that_are_not_finite(D, P, which, bad):
    gen = torch.Generator(device=DEV).manual_seed(D)
    H, T = 2, 130
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=gen)
    x = dict(r=rnd(T, H * D), k=rnd(T, H * D), v=rnd(T, H * P), w=torch.exp(-torch.exp(rnd(T, H * D) - 1)))
    gate, u, norm = rnd(T, H * P).to(torch.bfloat16), rnd(H * D), 1 + 0.1 * rnd(H * P)
    cu, slots = torch.tensor([0, T], dtype=torch.int32, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    chunks = ops().decay_chunks_of([T])

    def run(x):
        out, state = torch.empty(T, H * P, device=DEV, dtype=torch.bfloat16), torch.zeros(1, ops().decay_state_floats(H, D, P), device=DEV)
        ops().decay_chunks((x["r"], 0), (x["k"], 0), (x["v"], 0), (x["w"], 0), u, state, 0, cu, slots, chunks,
                           torch.empty(ops().decay_chunk_floats(chunks, H, D, P), device=DEV), gate, 0, norm, 1e-5, out, H, D, P)
        return out

    clean = run(x)
    for s in (1, 2, 3, 30, 36, 61, 63, 67, 129):
        spoilt = dict(x, **{which: x[which].clone()})
        spoilt[which][s] = bad
        got = run(spoilt)
        first = s + 1 if which == "w" else s             # (a token's decay acts behind it)
        assert torch.equal(got[:first], clean[:first]), s
        assert first >= T or bool(got[first:].isnan().any()), s


# one token a request, heads of every number of lanes, a request without a token and one with two (left alone)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("H,D,P", [(1, 4, 4), (2, 8, 128), (2, 12, 20), (3, 64, 64), (2, 100, 68), (2, 128, 128)])
def test_decay_step(H, D, P, dtype):
    gen = torch.Generator(device=DEV).manual_seed(D + P)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=gen)
    lengths, eps = [1, 0, 1, 2, 1], 1e-5
    lengths = lengths + [0, 0]                           # padding: its rows lie behind the last token's
    T, B = sum(lengths) + 2, len(lengths)
    cu = torch.tensor([sum(lengths[:i]) for i in range(B + 1)], dtype=torch.int32, device=DEV)
    slots = torch.tensor([4, 3, 0, 2, 1, 0, 0], dtype=torch.int32, device=DEV)
    u, norm = rnd(H * D), 1 + 0.1 * rnd(H * P)
    state = torch.zeros(B, ops().decay_state_floats(H, D, P) + 4, device=DEV)
    r, k, v, w = rnd(T, H * D + 4), rnd(T, H * D), rnd(T, H * P), torch.rand(T, H * D, device=DEV, generator=gen)
    gate = rnd(T, H * P + 8).to(dtype)
    o = torch.empty(T, H * P, device=DEV)
    for _ in range(2):                                   # a state that is not zero, then the step beside the walk
        out = torch.full((T, H * P), float("nan"), device=DEV, dtype=dtype)
        walked = state.clone()
        scan = (r, 4), (k, 0), (v, 0), (w, 0), u
        ops().decay_scan(*scan, walked, 4, cu, slots, o, H, D, P)
        ops().decay_step(*scan, state, 4, cu, slots, gate, 8, norm, eps, out, H, D, P)
        for b, n in enumerate(lengths):
            row, st = int(cu[b]), int(slots[b])
            if b >= T - 2:
                assert not out[b].any()
                continue
            if n != 1:
                assert out[row:row + n].isnan().all()
                continue
            assert float((state[st] - walked[st]).abs().max()) <= 2.0 ** -22 * float(walked[st].abs().max() + 1)      # two roundings
            y = o[row].double().view(H, P)
            y = y / torch.sqrt((y * y).mean(-1, keepdim=True) + eps) * norm.double().view(H, P)
            y = y * torch.nn.functional.silu(gate[row, 8:].double().view(H, P))
            assert float((out[row].double().view(H, P) - y).norm() / y.norm()) <= (2.0 ** -8 if dtype == torch.bfloat16 else 1e-6)
        state = walked


def state_of(flat, H, D, P):
    """decay_scan's state of one request as [H, D, P] in float64."""
    rows, lanes, cols, tiles = ops().decay_scan_shape(D, P)
    x = flat.double().view(H, tiles, rows, cols, lanes)              # element (row l rows + i, column z cols + col)
    return x.permute(0, 4, 2, 1, 3).reshape(H, lanes * rows, tiles * cols)[:, :D, :P]


# the float32 kernel of one token and head: fewer keys than groups, whole and broken pages, windows, kept keys, heads on both sides of 128
@pytest.mark.parametrize("hd", [16, 128, 144])
@pytest.mark.parametrize("page,window,keep", [(4, None, None), (16, 5, 3), (64, 40, 17)])
def test_paged_attention_reads_ahead(hd, page, window, keep):
    nq, nkv, lengths, scale = 4, 2, [1, 15, 16, 17, 33, 100, 64], hd ** -0.5
    T, blocks = len(lengths), -(-max(lengths) // page)
    gen = torch.Generator(device=DEV).manual_seed(hd + page)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=gen)
    table = torch.randperm(T * blocks, device=DEV, generator=gen).to(torch.int32).view(T, blocks)
    kc, vc, qkv = rnd(T * blocks, nkv, page, hd), rnd(T * blocks, nkv, page, hd), rnd(T, (nq + 2 * nkv) * hd)
    for t, n in enumerate(lengths):                      # pages wholly behind a request's last key or between kept keys and window are gone
        for b in range(blocks):
            if b * page >= n or (window and (b + 1) * page <= n - window and b * page >= keep):
                table[t, b] = -1
    pos, req = torch.tensor([n - 1 for n in lengths], dtype=torch.int32, device=DEV), torch.arange(T, dtype=torch.int32, device=DEV)
    out, err = torch.empty(T, nq * hd, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    ops().paged_attention(qkv, out, kc, vc, table, req, pos, nq, nkv, hd, scale, window, err, keep=keep)
    assert int(err) == 0
    for t, n in enumerate(lengths):
        j = torch.arange(n, device=DEV)
        seen = (j >= n - window) | (j < keep) if window else j >= 0
        rows = lambda c: c[table[t].clamp(min=0).long()].double().transpose(0, 1).reshape(nkv, -1, hd)[:, :n].repeat_interleave(nq // nkv, 0)
        s = torch.einsum("hd,hnd->hn", qkv[t, :nq * hd].double().view(nq, hd), rows(kc)) * scale
        ref = torch.einsum("hn,hnd->hd", torch.softmax(s.masked_fill(~seen, float("-inf")), -1), rows(vc))
        assert float((out[t].double().view(nq, hd) - ref).abs().max()) <= 1e-5 * float(ref.abs().max())      # float32 sums of up to 100 terms


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("hd", [16, 64, 96, 128, 144])
@pytest.mark.parametrize("weighting,window", [("softmax", None), ("softmax", 40), ("sigmoid", None)])
def test_paged_attention_holds_the_same_bits_for_few_and_for_many_tokens(hd, dtype, weighting, window):
    """Few blocks read a key ahead, many do not: the arithmetic is the same, and a token's bits depend on its positions alone."""
    nq, nkv, lengths, page = 4, 2, [1, 15, 16, 17, 33, 100, 64], 16
    n, blocks = len(lengths), -(-max(lengths) // page)
    gen = torch.Generator(device=DEV).manual_seed(hd)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=gen).to(dtype)
    table = torch.randperm(n * blocks, device=DEV, generator=gen).to(torch.int32).view(n, blocks)
    kc, vc, qkv = rnd(n * blocks, nkv, page, hd), rnd(n * blocks, nkv, page, hd), rnd(n, (nq + 2 * nkv) * hd)
    bias = torch.randn(nq, device=DEV, generator=gen) if weighting == "sigmoid" else None

    def run(times):
        pos = torch.tensor([m - 1 for m in lengths] * times, dtype=torch.int32, device=DEV)
        req = torch.arange(n, dtype=torch.int32, device=DEV).repeat(times)
        out, err = torch.empty(n * times, nq * hd, device=DEV, dtype=dtype), torch.zeros(1, dtype=torch.int32, device=DEV)
        ops().paged_attention(qkv.repeat(times, 1), out, kc, vc, table, req, pos, nq, nkv, hd, hd ** -0.5, window, err,
                              weighting=weighting, head_bias=bias)
        assert int(err) == 0
        return out.view(times, n, nq * hd)

    few = run(1)
    for times in (21, 22, 37, 38):                       # 588 and 616 blocks, 1,036 and 1,064
        assert bool((run(times) == few).all()), times


# the merge of a token's chunks: one, a batch of 128, more than one batch; chunks without keys in between, whose parts may hold anything; a window
# that begins behind some chunks; padding; sinks; columns of one thread's five and the rest
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("S", [1, 8, 127, 128, 129, 256, 300])
@pytest.mark.parametrize("hd,window,sink", [(16, None, False), (128, 2100, True), (576, None, True), (640, 500, False)])
def test_merge_of_chunks(S, hd, window, sink, dtype):
    nq, chunk, gen = 3, 16, torch.Generator(device=DEV).manual_seed(S + hd)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=gen)
    last = [S * chunk - 1, 0, -1, S * chunk // 2, max(S * chunk - 17, 0)]
    T = len(last)
    acc, ml = rnd(T, nq, S, hd), torch.stack([3 * rnd(T, nq, S), rnd(T, nq, S).abs() + 0.1], -1)
    empty = rnd(T, nq, S) < -1
    for t, p in enumerate(last):                         # chunks behind the last key or before the window are never read
        lo = max(0, p - window + 1) if window else 0
        empty[t, :, p // chunk if p >= 0 else 0] = False
        out_of_reach = torch.ones(S, dtype=torch.bool, device=DEV)
        out_of_reach[lo // chunk:p // chunk + 1] = p < 0
        acc[t][:, out_of_reach], ml[t][:, out_of_reach] = float("nan"), float("nan")
    inside = ~ml[..., 0].isnan() & empty
    ml[..., 0][inside] = float("-inf")
    ml[..., 1][inside], acc[inside] = float("nan"), float("nan")
    pos = torch.tensor(last, dtype=torch.int32, device=DEV)
    sinks = rnd(nq) if sink else None
    out = torch.full((T, nq * hd), 7.0, device=DEV, dtype=dtype)
    o = ops()
    o._check(o._fn("attention", "vl_decode_attention_merge")(acc.data_ptr(), ml.data_ptr(), pos.data_ptr(), out.data_ptr(), o.dtype_code(dtype), T, nq, hd,
                                                             chunk, S, window or 0, None, sinks.data_ptr() if sink else None, o._stream()), "merge")
    m = torch.where(ml[..., 0].isnan(), float("-inf"), ml[..., 0].double())
    top = m.max(-1, keepdim=True).values.clamp(min=-1e30)
    w = torch.exp(m - top)
    parts = torch.where((w > 0)[..., None], acc.double(), 0.0)
    total = (w * torch.where(w > 0, ml[..., 1].double(), 0.0)).sum(-1)
    if sink:
        total = total + torch.exp(sinks.double() - top[..., 0])
    live = torch.tensor([p >= 0 for p in last], device=DEV)[:, None, None]
    ref = torch.where(live, (w[..., None] * parts).sum(2) / total[..., None], 0.0)
    size = torch.where(live, (w[..., None] * parts.abs()).sum(2) / total[..., None], 0.0)
    # S roundings of float32 sums, weights good to 2^-20 (bfloat16: the fast exponential), the output's rounding
    rel = (S + 8) * 2.0 ** -24 + 2.0 ** -20
    got = out.double().view(T, nq, hd)
    assert bool(((got - ref).abs() <= rel * size + (2.0 ** -8 if dtype == torch.bfloat16 else 0) * ref.abs()).all())


# the few-row product of routed experts: items of one block and of several, more items than places, places without rows in between,
# padding rows, K at a step's edge and not, N at a tile's edge and not
@pytest.mark.parametrize("N,K", [(16, 512), (144, 520), (4096, 1024), (8192, 2048)])
@pytest.mark.parametrize("groups", [[0], [2, 2, 0, 1], [1, -1, 0, -1, -1, 2, -1], [-1, -1], list(range(3)) * 7 + [-1] * 4])
@pytest.mark.parametrize("act", [None, "silu"])
def test_experts_product_of_few_rows(groups, N, K, act):
    gen = torch.Generator(device=DEV).manual_seed(N + K + len(groups))
    top, tokens, cap = 2, 24, 16 * len(groups)
    h = torch.randn(tokens, K, device=DEV, generator=gen).to(torch.bfloat16)
    w = (torch.randn(3, N, K, device=DEV, generator=gen) / K ** 0.5).to(torch.bfloat16)
    rows = torch.randint(-8, tokens * top, (cap,), device=DEV, generator=gen).clamp(min=-1).to(torch.int32)      # pair or -1
    scale = torch.rand(tokens * top, device=DEV, generator=gen)
    tile_group = torch.tensor(groups, dtype=torch.int32, device=DEV)
    out = torch.full((cap, N // 2 if act else N), 7.0, device=DEV, dtype=torch.bfloat16)
    ops().gemm_grouped_fused(h, w, out, tile_group, 16, rows, top, scale, act, 1.0, 0.0, 0.0)
    for y, e in enumerate(groups):
        at = slice(16 * y, 16 * y + 16)
        if e < 0:
            assert bool((out[at] == 7.0).all())          # a place without rows is left alone
            continue
        r = rows[at].long()
        a = h.double()[r.clamp(min=0) // top] * (r >= 0)[:, None]
        s = torch.where(r >= 0, scale.double()[r.clamp(min=0)], 0.0)[:, None]
        z, size = (a @ w[e].double().T) * s, (a.abs() @ w[e].double().abs().T) * s
        off = K * 2.0 ** -24 * size                      # float32 sums
        if act:
            z, off = z.view(16, -1, 2, 8), off.view(16, -1, 2, 8)
            g, u = z[:, :, 0].reshape(16, -1), z[:, :, 1].reshape(16, -1)
            og, ou = off[:, :, 0].reshape(16, -1), off[:, :, 1].reshape(16, -1)
            z, off = g / (1 + torch.exp(-g)) * u, 1.2 * og * u.abs() + g.abs() * ou
        assert bool(((out[at].double() - z).abs() <= 2.0 ** -8 * z.abs() + off + 1e-6).all())
    if act is None:                                      # the same rows without the index, as the second product takes them
        sorted_rows = h[rows.clamp(min=0).long() // top].contiguous()
        again = torch.full((cap, N), 7.0, device=DEV, dtype=torch.bfloat16)
        ops().gemm_grouped(sorted_rows, w, again, tile_group, 16)
        live = (tile_group >= 0).repeat_interleave(16) & (rows >= 0)
        ref = torch.stack([sorted_rows[m].double() @ w[groups[m // 16]].double().T for m in range(cap) if live[m]]) if bool(live.any()) else again[live].double()
        assert bool(((again[live].double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-3).all())


# ... and where two blocks an SM would need a second round and three do not (a ring of three stages): the first and the last number of items of
# that range, K of fewer stages than the ring's and of several rounds of it, cut at the end; every activation
@pytest.mark.parametrize("act", [None, "silu", "relu", "capped_swish", "relu2"])
@pytest.mark.parametrize("K", [512, 1160])
@pytest.mark.parametrize("last,dead", [(False, 0), (True, 0), (True, 2)])
def test_experts_product_of_few_rows_in_one_round_of_three_blocks(last, dead, K, act):
    sms = 2 * ops().sm_pairs()
    N, G, top, tokens = 64 * 12, 5, 2, 40
    across, gated = N // 64, act in ("silu", "relu", "capped_swish")
    tiles = 3 * sms // across if last else 2 * sms // across + 1
    assert 2 * sms < tiles * across <= 3 * sms                     # the launcher's items: of all places, rows or none
    groups = [y % G for y in range(tiles - dead)] + [-1] * dead
    gen = torch.Generator(device=DEV).manual_seed(K + tiles)
    cap = 16 * tiles
    h = torch.randn(tokens, K, device=DEV, generator=gen).to(torch.bfloat16)
    w = (torch.randn(G, N, K, device=DEV, generator=gen) / K ** 0.5).to(torch.bfloat16)
    rows = torch.randint(-8, tokens * top, (cap,), device=DEV, generator=gen).clamp(min=-1).to(torch.int32)
    scale, err = torch.rand(tokens * top, device=DEV, generator=gen), torch.zeros(1, dtype=torch.int32, device=DEV)
    out = torch.full((cap, N // 2 if gated else N), 7.0, device=DEV, dtype=torch.bfloat16)
    ops().gemm_grouped_fused(h, w, out, torch.tensor(groups, dtype=torch.int32, device=DEV), 16, rows, top, scale, act, 1.5, 0.8, 0.25, err)
    assert int(err) == 0
    for y, e in enumerate(groups):
        at = slice(16 * y, 16 * y + 16)
        if e < 0:
            assert bool((out[at] == 7.0).all())
            continue
        r = rows[at].long()
        a = h.double()[r.clamp(min=0) // top] * (r >= 0)[:, None]
        s = torch.where(r >= 0, scale.double()[r.clamp(min=0)], 0.0)[:, None]
        z, off = (a @ w[e].double().T) * s, K * 2.0 ** -24 * (a.abs() @ w[e].double().abs().T) * s          # float32 sums
        if gated:
            z, off = z.view(16, -1, 2, 8), off.view(16, -1, 2, 8)
            p, u, op, ou = z[:, :, 0].reshape(16, -1), z[:, :, 1].reshape(16, -1), off[:, :, 0].reshape(16, -1), off[:, :, 1].reshape(16, -1)
            if act == "relu":
                z, off = p.clamp(min=0) * u, op * u.abs() + p.abs() * ou + op * ou
            else:
                alpha, shift = 1.0, 0.0
                if act == "capped_swish":
                    alpha, shift, p, u = 1.5, 0.25, p.clamp(max=0.8), u.clamp(-0.8, 0.8)
                z = p / (1 + torch.exp(-alpha * p)) * (u + shift)          # |d/dp p sigmoid(alpha p)| <= 1.1
                off = 1.2 * op * (u + shift).abs() + p.abs() * ou + 2.0 ** -20 * z.abs()
        elif act == "relu2":
            off = 2 * z.abs() * off + off * off
            z = z.clamp(min=0) ** 2
        assert bool(((out[at].double() - z).abs() <= 2.0 ** -8 * z.abs() + off + 1e-6).all()), y


# the batched product of many rows: results that leave 16 bytes, two numbers and one number at a time, by the rows' alignment; tiles cut in rows and
# columns; with an output gate (bfloat16)
@pytest.mark.parametrize("H,N", [(2, 104), (2, 98), (3, 97), (1, 130), (2, 257)])
@pytest.mark.parametrize("T", [512, 700])
@pytest.mark.parametrize("out_dtype,gated", [(torch.bfloat16, False), (torch.bfloat16, True), (torch.float32, False)])
def test_products_per_head_of_many_rows(T, H, N, out_dtype, gated):
    K, gen = 136, torch.Generator(device=DEV).manual_seed(T + H * N)
    a = torch.randn(T, H * K, device=DEV, generator=gen).to(torch.bfloat16)
    w = (torch.randn(H, N, K, device=DEV, generator=gen) / K ** 0.5).to(torch.bfloat16)
    gate = torch.randn(T, H, device=DEV, generator=gen).to(torch.bfloat16)
    out = torch.full((T + 1, H * N), 7.0, device=DEV, dtype=out_dtype)
    ops().gemm_heads(a, w, out[:T], **(dict(gate=gate) if gated else {}))
    x, v = a.double().view(T, H, K), w.double()
    ref, size = torch.einsum("thk,hnk->thn", x, v), torch.einsum("thk,hnk->thn", x.abs(), v.abs())
    if gated:
        ref, size = ref * torch.sigmoid(gate.double())[:, :, None], size * torch.sigmoid(gate.double())[:, :, None]
    bound = (K + 8) * 2.0 ** -24 * size + (2.0 ** -8 * ref.abs() if out_dtype == torch.bfloat16 else 0)
    assert bool(((out[:T].double().view(T, H, N) - ref).abs() <= bound).all()) and bool((out[T:] == 7.0).all())


@pytest.mark.parametrize("H", [96, 1028, 2048, 4096, 8192])
@pytest.mark.parametrize("act", [torch.float32, torch.bfloat16])
def test_norms_of_few_and_of_many_rows_hold_the_same_bits(H, act):
    """Few rows read weights and stream ahead of the row's sum, many rows behind it: same arithmetic, so a row's bits do not depend on how many
    rows there are.  593 rows never read ahead; 592 and 444 are the last that do (bfloat16, float32), 296 for rows beyond 4,096, and one
    norm does so while a kernel before it drains."""
    from vllm_lite_b200.parts.base import StreamSum
    R = 593
    g = torch.Generator(device=DEV).manual_seed(H)
    x, w = torch.randn(R, H, generator=g, device=DEV), torch.randn(H, generator=g, device=DEV)
    y = torch.randn(R, H, generator=g, device=DEV).to(act)

    def run(rows, pdl=False):
        a, b, c = x[:rows].clone(), x[:rows].clone(), x[:rows].clone()
        delta, out = y[:rows].contiguous(), torch.empty(rows, H, device=DEV, dtype=act)
        normed = torch.empty_like(out)
        ops().set_pdl(pdl)
        try:
            ops().add_rmsnorm(a, delta, w, 1e-6, out)
            ops().rmsnorm_add(delta, w, 1e-6, 0.5, b)
            ops().stream_norm(c, StreamSum(a=delta, a_scale=w, mult=0.5), w, 1e-6, normed)
        finally:
            ops().set_pdl(False)
        return a, out, b, c, normed

    many = run(R)
    for rows, pdl in ((592, False), (445, False), (444, False), (297, False), (296, False), (1, False), (64, True), (296, True)):
        for f, m in zip(run(rows, pdl), many):
            assert torch.equal(f, m[:rows]), (rows, pdl)
    add = x + y.float()
    # float32: 32 running additions a thread and 8 levels of tree leave at most 40 2^-24 on the sum, half of it on the root, and a few products
    want = add * torch.rsqrt(add.double().pow(2).mean(-1, keepdim=True) + 1e-6).float() * w
    assert (many[1].float() - want).abs().max() < (2 ** -8 if act == torch.bfloat16 else 2 ** -18) * want.abs().max()


# a residual of float32 sums beside bfloat16 rows: x + delta is one float32 addition, vectorised, by eights and one by one
@pytest.mark.parametrize("H", [96, 1030, 4096, 16384])
@pytest.mark.parametrize("rows", [1, 12, 700])
def test_norm_adds_float32_sums(H, rows):
    g = torch.Generator(device=DEV).manual_seed(H + rows)
    x, d, w = (torch.randn(n, generator=g, device=DEV) for n in ((rows, H), (rows, H), (H,)))
    a, out = x.clone(), torch.empty(rows, H, device=DEV, dtype=torch.bfloat16)
    ops().add_rmsnorm(a, d, w, 1e-6, out)
    assert torch.equal(a, x + d)
    b, same = a.clone(), torch.empty_like(out)
    ops().add_rmsnorm(b, None, w, 1e-6, same)                                 # the norm of the stream that the addition left
    assert torch.equal(same, out) and torch.equal(a, b)
    pick = torch.tensor([rows - 1, 0], dtype=torch.int32, device=DEV)
    few, c = torch.empty(2, H, device=DEV, dtype=torch.bfloat16), x.clone()
    ops().add_rmsnorm(c, d, w, 1e-6, few, rows=pick)
    assert torch.equal(few, out[pick.long()]) and torch.equal(c, x)


# the router's product on tiles of 16 and of 64 rows: a row's bits do not depend on how many rows there are (the taller tiles begin at 1,536 rows of
# eight parts of K, 3,009 of four, 12,225 of one, with up to 64 columns), remainders in rows and columns
@pytest.mark.parametrize("K,N,sizes", [(2048, 32, (1535, 1536, 1537)), (1024, 40, (3008, 3009, 3073)), (264, 8, (12224, 12225)), (1024, 130, (1535, 1536, 1600))])
def test_router_product_holds_the_same_bits_on_both_tiles(K, N, sizes):
    gen = torch.Generator(device=DEV).manual_seed(K)
    h = torch.randn(sizes[-1], K, device=DEV, generator=gen).to(torch.bfloat16)
    router, parts = torch.randn(N, K, device=DEV, generator=gen).to(torch.bfloat16), ops().router_slices(K)

    def run(rows):
        sums = torch.full((parts, rows, N), float("nan"), device=DEV)
        ids, w = torch.empty(rows, 1, dtype=torch.int32, device=DEV), torch.empty(rows, 1, device=DEV)
        ops().moe_route(h[:rows], router, 1, ids, w, sums)
        return sums

    few = run(16)
    for rows in sizes:
        sums = run(rows)
        assert torch.equal(sums[:, :16], few)
        # (another tile's remainder: the last rows by themselves)
        assert torch.equal(sums[:, rows - 1], run_rows(h[rows - 1:rows], router, parts))
        ref, size = h[:rows].double() @ router.double().T, h[:rows].double().abs() @ router.double().abs().T
        assert bool(((sums.double().sum(0) - ref).abs() <= K * 2.0 ** -24 * size).all())      # K roundings of sums that stay below it


def run_rows(h, router, parts):
    sums = torch.empty(parts, h.shape[0], router.shape[0], device=DEV)
    ops().moe_route(h.contiguous(), router, 1, torch.empty(h.shape[0], 1, dtype=torch.int32, device=DEV), torch.empty(h.shape[0], 1, device=DEV), sums)
    return sums[:, 0]


def test_a_row_of_nan_is_routed_to_experts_that_exist():
    T, K, E, top = 5, 64, 40, 4
    gen = torch.Generator(device=DEV).manual_seed(5)
    h, router = torch.randn(T, K, device=DEV, generator=gen), torch.randn(E, K, device=DEV, generator=gen)
    h[2] = float("nan")
    ids, w = torch.full((T, top), -1, dtype=torch.int32, device=DEV), torch.empty(T, top, device=DEV)
    ops().moe_route(h, router, top, ids, w, torch.empty(ops().router_slices(K), T, E, device=DEV))
    assert bool(((ids >= 0) & (ids < E)).all()) and bool(w[2].isnan().any())     # (and the NaN goes on)
    good = [0, 1, 3, 4]
    assert torch.equal(ids[good].long(), (h.double() @ router.double().T)[good].topk(top).indices)


@pytest.mark.parametrize("H,offset", [(1, 0), (96, 0), (96, 1), (1024, 0), (1028, 0), (4100, 0), (4101, 0)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_embedding_rows(H, offset, dtype):
    V, ids = 50, torch.tensor([0, 49, 7, -1, 50, 7], dtype=torch.int32, device=DEV)
    table = torch.randn(V * H + offset, device=DEV).to(dtype)[offset:].view(V, H)     # offset: rows off the 16-byte boundary
    out, err = torch.full((6, H), float("nan"), device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    ops().embed(ids, table, out, err, 3.0)
    want = table.float()[ids.long().clamp(0, V - 1)] * 3.0
    want[3:5] = 0
    assert torch.equal(out, want) and int(err) != 0


# the many-row product of routed experts: groups without rows, of less than a tile, at its edges and of several; fewer tiles than
# pairs of SMs and more; N below, at and beside a tile's edge, K with a short last block
@pytest.mark.parametrize("sizes", [[0, 16, 0, 256, 272, 0], [32, 240, 256, 16, 48], [700, 0, 1333, 5], [3] * 40, [0, 0, 2048]])
@pytest.mark.parametrize("N,K", [(16, 72), (192, 1096), (512, 2048), (2064, 520)])
@pytest.mark.parametrize("act", [None, "silu", "relu", "capped_swish", "relu2"])
def test_experts_product_of_many_rows(sizes, N, K, act):
    G = len(sizes)
    gen = torch.Generator(device=DEV).manual_seed(N + K + sum(sizes))
    starts = [0]
    for n in sizes:
        starts.append(starts[-1] + -(-n // 16) * 16)
    cap = starts[-1] + 32                                # rows behind the last group, which nobody writes
    rows = torch.randn(cap, K, device=DEV, generator=gen).to(torch.bfloat16)
    w = (torch.randn(G, N, K, device=DEV, generator=gen) / K ** 0.5).to(torch.bfloat16)
    scale = torch.rand(cap, device=DEV, generator=gen) if act == "silu" else None
    index = torch.randperm(cap, device=DEV, generator=gen).to(torch.int32) if act == "silu" else None
    gated = act in ("silu", "relu", "capped_swish")
    e = torch.zeros(1, dtype=torch.int32, device=DEV)
    start_rows = torch.tensor(starts, dtype=torch.int32, device=DEV)
    outs = []
    for _ in range(2):
        out = torch.full((cap, N // 2 if gated else N), 7.0, device=DEV, dtype=torch.bfloat16)
        ops().gemm_grouped_tc5(rows, w, out, start_rows, e, index, scale, act, 1.5, 0.8, 0.25)
        outs.append(out)
    assert int(e.item()) == 0 and torch.equal(outs[0], outs[1])
    assert bool((outs[0][starts[-1]:] == 7.0).all())
    for g in (g for g in range(G) if sizes[g]):
        at = slice(starts[g], starts[g + 1])
        s = scale.double()[index[at].long()][:, None] if scale is not None else 1.0
        z = (rows[at].double() @ w[g].double().T) * s
        off = K * 2.0 ** -24 * (rows[at].double().abs() @ w[g].double().abs().T) * s        # float32 sums
        if gated:
            z, off = z.view(z.shape[0], -1, 2, 8), off.view(z.shape[0], -1, 2, 8)
            p, u = z[:, :, 0].reshape(z.shape[0], -1), z[:, :, 1].reshape(z.shape[0], -1)
            op, ou = off[:, :, 0].reshape(z.shape[0], -1), off[:, :, 1].reshape(z.shape[0], -1)
            if act == "relu":
                z, off = p.clamp(min=0) * u, op * u.abs() + p.abs() * ou + op * ou
            else:
                a, shift = 1.0, 0.0
                if act == "capped_swish":
                    a, shift, p, u = 1.5, 0.25, p.clamp(max=0.8), u.clamp(-0.8, 0.8)
                # |d/dp p sigmoid(a p)| <= 1.1; sigmoid by the fast exponential and a division: a few roundings
                z, off = p / (1 + torch.exp(-a * p)) * (u + shift), 1.2 * op * (u + shift).abs() + p.abs() * ou + 2.0 ** -20 * (p * (u + shift)).abs()
        elif act == "relu2":
            off = 2 * z.abs() * off + off * off
            z = z.clamp(min=0) ** 2
        assert bool(((outs[0][at].double() - z).abs() <= 2.0 ** -8 * z.abs() + off + 1e-6).all()), g


@pytest.mark.parametrize("act", ["silu", "capped_swish"])
def test_experts_product_with_the_full_exponential(act):
    """Gates of -20 to -75 and ups of 1, both exact sums: what is rounded is the activation alone.  A float32 activation (exponential to 1 ulp, sum,
    quotient: 4 x 2^-24 at most) rounds to another bfloat16 number than the exact one where it crosses the middle of a step of 2^-8 or
    more: 6.1e-5 of the results at most.  The fast exponential, whose argument of up to 108 is rounded to 2^-18, crosses three times as many."""
    M, K, pairs = 16384, 64, 128
    gen = torch.Generator(device=DEV).manual_seed(4)
    rows = torch.zeros(M, K, device=DEV)
    rows[:, 0] = -20 - 30 * torch.rand(M, device=DEV, generator=gen)
    rows[:, 1], rows[:, 2] = 1.0, torch.rand(M, device=DEV, generator=gen) / 2      # (what makes every gate another one)
    rows[:, 2] = (rows[:, 2] * 2 ** 9).round() / 2 ** 9
    rows = rows.to(torch.bfloat16)
    w = torch.zeros(1, 2 * pairs, K, device=DEV)
    fine = 1 + torch.arange(pairs, device=DEV) / 256.0                       # gates: rows[:, 0] times these, products of two 8-bit numbers
    w.view(-1, 2, 8, K)[:, 0, :, 0], w.view(-1, 2, 8, K)[:, 0, :, 2], w.view(-1, 2, 8, K)[:, 1, :, 1] = fine.to(torch.bfloat16).float().view(-1, 8), 1.0, 1.0
    err, out = torch.zeros(1, dtype=torch.int32, device=DEV), torch.empty(M, pairs, device=DEV, dtype=torch.bfloat16)
    starts = torch.tensor([0, M], dtype=torch.int32, device=DEV)
    ops().gemm_grouped_tc5(rows, w.to(torch.bfloat16), out, starts, err, act=act, alpha=1.0, limit=1e9, shift=0.0, fine=True)
    g = rows[:, :1].double() * fine.to(torch.bfloat16).double() + rows[:, 2:3].double()
    exact = (g / (1 + torch.exp(-g))).float()                                # (one rounding to float32 first: 2^-15 of a bfloat16 step)
    assert float((out != exact.to(torch.bfloat16)).float().mean()) <= 6.1e-5 and int(err) == 0


# functions of one argument: eight, four and single values a thread, and buffers that begin anywhere
@pytest.mark.parametrize("act", ["gelu", "tanh", "relu2"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n,off", [(1, 0), (7, 0), (12, 0), (148 * 2048 - 8, 0), (148 * 2048, 0), (148 * 2048 + 4, 0), (4096, 1)])
def test_unary_activation(act, dtype, n, off):
    gen = torch.Generator(device=DEV).manual_seed(n)
    x = (3 * torch.randn(n + off, device=DEV, generator=gen)).to(dtype)[off:]
    x[: min(n, 5)] = torch.tensor([0.0, -12.9, 13.1, -0.0, 1e-30], device=DEV, dtype=dtype)[: min(n, 5)]
    out = torch.full((n + off,), 7.0, device=DEV, dtype=dtype)[off:]
    ops().unary_act(x, out, act)
    v = x.double()
    ref = v * 0.5 * torch.special.erfc(-v / 2 ** 0.5) if act == "gelu" else torch.tanh(v) if act == "tanh" else v.clamp(min=0) ** 2
    # gelu in float32: the exponent z^2 (up to 85 here) carries a rounding of 2^-23, the polynomial 2^-22, the rest a few roundings
    rel = (85 + 8) * 2.0 ** -23 + (2.0 ** -8 if dtype == torch.bfloat16 else 0)
    assert bool(((out.double() - ref).abs() <= rel * ref.abs() + 1e-37).all())


def test_gelu_of_small_float32_values():
    """|v| <= 0.5: 1 + erff(z) to 2 ulp of erff (2^-24 here), 0.6 of that for the rounded argument and the sum's own 2^-24, relative to a sum of
    0.61 or more, then a product.  And the same bits whether or not neighbours lie on the other side of -1.5, where the form changes."""
    x = torch.linspace(-0.5, 0.5, 200_001, device=DEV)
    x = x[x != 0]
    out = ops().unary_act(x, torch.empty_like(x), "gelu")
    ref = x.double() * 0.5 * torch.special.erfc(-x.double() / 2 ** 0.5)
    assert bool(((out.double() - ref).abs() <= 6.2 * 2.0 ** -24 * ref.abs()).all())
    both = torch.stack([x[:1000], x[:1000] - 3], 1).reshape(-1).contiguous()
    assert torch.equal(ops().unary_act(both, torch.empty_like(both), "gelu")[::2], out[:1000])


def test_gelu_of_bfloat16_values_is_that_of_float32_rounded_once():
    gen = torch.Generator(device=DEV).manual_seed(2)
    x = torch.randn(1 << 20, device=DEV, generator=gen).clamp(min=-1.49).to(torch.bfloat16)
    wide = ops().unary_act(x.float(), torch.empty(x.shape, device=DEV), "gelu")
    assert torch.equal(ops().unary_act(x, torch.empty_like(x), "gelu"), wide.to(torch.bfloat16))


def test_gelu_beyond_numbers():
    x = torch.tensor([float("inf"), float("nan"), 3e38, -3e38], device=DEV)
    out = torch.empty_like(x)
    ops().unary_act(x, out, "gelu")
    got = out.tolist()
    assert got[0] == float("inf") and got[1] != got[1] and got[2] == x[2].item() and got[3] == 0.0
