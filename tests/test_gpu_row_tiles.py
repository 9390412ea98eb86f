"""Row-wise tiles on their own, in the fabric: tiles whose rows stream through the operand ring and tiles of few rows, at the
edges of both, against the same formulas in 64 bits or, where the result's bits are defined, against one another."""
import numpy as np
import pytest
import torch

from monoserve_b200.fabric import Program, Tile
from monoserve_b200.fabric.args import pack
from tests.test_gpu_fabric_gemm import fab, run_program  # noqa: F401

pytestmark = pytest.mark.gpu

K_STREAMS, K_RESIDUAL = 53, 66
EPS = 1e-5


def run_rows(fab, kind, block, rows, per):  # noqa: F811
    args = torch.frombuffer(bytearray(block), dtype=torch.uint8).cuda()
    p = Program()
    tiles = [Tile(kind, i=(r, min(per, rows - r)), a=(args.data_ptr(),)) for r in range(0, rows, per)]
    run_program(fab, p, p.stage(tiles))


def close(got, want, what):
    """fp32 sums of a few thousand terms: 2^-24 of each, some of them added in a row (32-bit outputs); bf16: 2^-9 a value."""
    limit = 4e-3 if got.dtype == torch.bfloat16 else 2e-6
    err = float((got.double() - want).norm() / want.norm())
    assert err < limit, (what, err)


def over_rms(x):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + EPS)


# rows of a tile: below and at the number that streams, more than the ring holds; the last tile of each is a short one.
# widths: one thread's columns, not a multiple of the block's, full, a ring of two or three rows, wider than the streamed form
@pytest.mark.parametrize("per", [3, 4, 29])
@pytest.mark.parametrize("W,ns,parts", [(4, 1, 1), (520, 3, 2), (2048, 4, 1), (2052, 4, 1), (4096, 4, 2), (4100, 2, 1), (2048, 4, 8)])
def test_streams(fab, W, ns, parts, per):  # noqa: F811
    g = torch.Generator(device="cuda").manual_seed(W + per)
    rows, slab = 2 * per + 5, 70
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    xs, y, w = r(rows, ns, W), r(parts, slab, W), 1 + 0.1 * r(W)
    h_in, h_out, mix = r(ns), r(ns), r(ns, ns)
    gather = torch.full((rows,), -1, dtype=torch.int32, device="cuda")
    gather[rows - 1], gather[0] = 0, 1
    h16, out16 = (torch.zeros(n, W, device="cuda", dtype=torch.bfloat16) for n in (rows, 2))
    h32, sum_out = torch.zeros(rows, W, device="cuda"), torch.zeros(rows, W, device="cuda")
    new = torch.einsum("su,rsw->ruw", mix.double(), xs.double()) + h_out.double()[None, :, None] * y.double().sum(0)[:rows, None]
    h = over_rms(torch.einsum("s,rsw->rw", h_in.double(), new)) * w.double()
    block = pack("StreamArgs", xs=xs, y=y, hc_out=h_out, hc_mix=mix, hc_in=h_in, w=w, h16=h16, h32=h32, gather=gather, out16=out16,
                 sum_out=sum_out, W=W, streams=ns, ld_h16=W, ld_h32=W, ld_out=W, y_parts=parts, y_rows=slab, eps=EPS)
    torch.cuda.synchronize()
    run_rows(fab, K_STREAMS, block, rows, per)
    close(xs, new, "streams")
    close(sum_out, new.sum(1), "sum")
    close(h32, h, "h32")
    close(h16, h, "h16")
    close(out16, h[[rows - 1, 0]], "gathered")


@pytest.mark.parametrize("per", [3, 4, 29])
@pytest.mark.parametrize("W,parts", [(4, (1, 0)), (520, (2, 1)), (2048, (1, 1)), (2052, (1, 0)), (4096, (1, 2)), (4100, (1, 0)), (2048, (8, 8))])
def test_residual(fab, W, parts, per):  # noqa: F811
    g = torch.Generator(device="cuda").manual_seed(W + per)
    rows, slab = 2 * per + 5, 70
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    x, y0, y1 = r(rows, W), r(parts[0], slab, W), r(max(1, parts[1]), slab, W)
    w, post, w0, w1 = (1 + 0.1 * r(W) for _ in range(4))
    gather = torch.full((rows,), -1, dtype=torch.int32, device="cuda")
    gather[rows - 1], gather[0] = 0, 1
    h16, out16 = (torch.zeros(n, W, device="cuda", dtype=torch.bfloat16) for n in (rows, 2))
    h32, sum_out = torch.zeros(rows, W, device="cuda"), torch.zeros(rows, W, device="cuda")
    y = y0.double().sum(0)[:rows]
    if parts[1]:
        y = 0.5 * (over_rms(y) * w0.double() + over_rms(y1.double().sum(0)[:rows]) * w1.double())
    new = x.double() + over_rms(y) * post.double()
    h = over_rms(new) * w.double()
    block = pack("ResidualArgs", x=x, y0=y0, y1=y1, post_w=post, w0=w0, w1=w1, w=w, h16=h16, h32=h32, gather=gather, out16=out16,
                 sum_out=sum_out, W=W, ld_h16=W, ld_h32=W, ld_out=W, y0_parts=parts[0], y1_parts=parts[1], y_rows=slab, eps=EPS,
                 branch_scale=0.5)
    torch.cuda.synchronize()
    run_rows(fab, K_RESIDUAL, block, rows, per)
    close(x, new, "residual")
    close(sum_out, new, "sum")
    close(h32, h, "h32")
    close(h16, h, "h16")
    close(out16, h[[rows - 1, 0]], "gathered")


@pytest.mark.parametrize("per", [3, 4, 29])
@pytest.mark.parametrize("W,ns", [(8, 1), (520, 3), (2048, 4), (2052, 4), (4096, 4), (4104, 2)])
def test_streams_embedding(fab, W, ns, per):  # noqa: F811
    g = torch.Generator(device="cuda").manual_seed(W + per)
    rows = 2 * per + 5
    embed, w, h_in = torch.randn(40, W, generator=g, device="cuda").to(torch.bfloat16), torch.randn(W, generator=g, device="cuda"), torch.rand(ns, device="cuda")
    tokens = torch.randint(0, 40, (rows,), generator=g, device="cuda", dtype=torch.int32)
    xs, h16 = torch.zeros(rows, ns, W, device="cuda"), torch.zeros(rows, W, device="cuda", dtype=torch.bfloat16)
    x = embed[tokens.long()].float()
    h = over_rms(x.double() * h_in.double().sum()) * w.double()
    block = pack("StreamArgs", xs=xs, hc_in=h_in, w=w, h16=h16, embed=embed, tokens=tokens, W=W, streams=ns, ld_h16=W, eps=EPS)
    torch.cuda.synchronize()
    run_rows(fab, K_STREAMS, block, rows, per)
    assert torch.equal(xs, x[:, None].expand(rows, ns, W))
    close(h16, h, "h16")


@pytest.mark.parametrize("positions", [True, False])
@pytest.mark.parametrize("per", [3, 4, 29])
@pytest.mark.parametrize("W", [8, 520, 2048, 2052, 4096, 4104])
def test_residual_embedding(fab, W, per, positions):  # noqa: F811
    g = torch.Generator(device="cuda").manual_seed(W + per)
    rows = 2 * per + 5
    embed, pos = (torch.randn(40, W, generator=g, device="cuda").to(torch.bfloat16) for _ in range(2))
    w = torch.randn(W, generator=g, device="cuda")
    tokens, at = (torch.randint(0, n, (rows,), generator=g, device="cuda", dtype=torch.int32) for n in (40, 50))   # positions past the table: its last row
    x, h16 = torch.zeros(rows, W, device="cuda"), torch.zeros(rows, W, device="cuda", dtype=torch.bfloat16)
    want = embed[tokens.long()].double() * 0.75
    if positions:
        want = want + pos[at.long().clamp(max=39)].double()
    block = pack("ResidualArgs", x=x, w=w, h16=h16, embed=embed, pos=pos if positions else 0, tokens=tokens, tok_pos=at, W=W, ld_h16=W,
                 embed_scale=0.75, max_pos=40, eps=EPS)
    torch.cuda.synchronize()
    run_rows(fab, K_RESIDUAL, block, rows, per)
    close(x, want, "residual")
    close(h16, over_rms(want) * w.double(), "h16")


@pytest.mark.parametrize("norm", [True, False])
@pytest.mark.parametrize("H,K,shared", [(256, 2, False), (512, 8, True), (768, 16, False), (2048, 8, False), (2048, 8, True), (4096, 8, True),
                                        (4352, 4, False)])
def test_combine_streamed_or_not(fab, H, K, shared, norm):  # noqa: F811
    """Tiles of 16 rows and more bring their rows through the ring; tiles of three do not: the same bits."""
    g = torch.Generator(device="cuda").manual_seed(H + K)
    rows = 2 * 29 + 17
    y = torch.randn(rows * K, H, generator=g, device="cuda")
    x2, w = (torch.randn(n, H, generator=g, device="cuda").to(torch.bfloat16) for n in (rows, 1))
    extra = torch.randn(rows, H, generator=g, device="cuda")
    tw = torch.rand(rows, K, generator=g, device="cuda")
    pos = torch.randperm(rows * K, generator=g, device="cuda").to(torch.int32)
    outs = []
    for per in (3, 29):
        x, out = (torch.zeros(rows, H, device="cuda", dtype=torch.bfloat16) for _ in range(2))
        block = pack("CombineArgs", y=y, pair_pos=pos, topk_w=tw, x2=x2, x=x, w=w if norm else 0, out=out, K=K, H=H, eps=EPS,
                     shared=extra if shared else 0)
        torch.cuda.synchronize()
        run_rows(fab, 47, block, rows, per)
        outs.append((x, out))
    for a, b in zip(*outs):
        assert torch.equal(a, b)
    want = x2.double() + (tw.double()[:, :, None] * y[pos.long()].double().view(rows, K, H)).sum(1) + (extra.double() if shared else 0)
    close(outs[0][0], want, "x")


@pytest.mark.parametrize("norm", [True, False])
@pytest.mark.parametrize("hq,hkv,rot", [(32, 4, 128), (6, 1, 64), (12, 2, 128), (2, 3, 0)])
def test_rope_of_eight_items_at_a_time(fab, hq, hkv, rot, norm):  # noqa: F811
    """Tiles whose warps take eight items of a row at a time and tiles that take one give the same bits."""
    g = torch.Generator(device="cuda").manual_seed(hq)
    rows, heads, page, pages = 37, hq + 2 * hkv, 16, 4
    qkv, wq, wk = (torch.randn(*s, generator=g, device="cuda").to(torch.bfloat16) for s in ((rows, heads * 128), (128,), (128,)))
    tok_pos = torch.randint(0, 50, (rows,), generator=g, device="cuda", dtype=torch.int32)
    tok_slot = torch.randperm(page * pages, generator=g, device="cuda")[:rows].to(torch.int32)
    cos_sin = torch.randn(40, max(1, rot // 2), 2, generator=g, device="cuda")   # 40 positions: further ones take the last
    outs = []
    for per in (24, 32, 96, rows * heads):
        q = torch.zeros(rows, hq, 128, device="cuda", dtype=torch.bfloat16)
        k, v = (torch.zeros(pages, page, hkv, 128, device="cuda", dtype=torch.bfloat16) for _ in range(2))
        block = pack("QkArgs", qkv=qkv, q_out=q, k_cache=k, v_cache=v, q_norm=wq if norm else 0, k_norm=wk if norm else 0, tok_pos=tok_pos,
                     tok_slot=tok_slot, cos_sin=cos_sin, ld_qkv=heads * 128, hq=hq, hkv=hkv, rot_dim=rot, eps=EPS, max_pos=40)
        torch.cuda.synchronize()
        run_rows(fab, 37, block, rows * heads, per)
        outs.append((q, k, v))
    for other in outs[1:]:
        for a, b in zip(outs[0], other):
            assert torch.equal(a, b)
    assert outs[0][2].view(-1, hkv, 128)[tok_slot.long()].equal(qkv.view(rows, heads, 128)[:, hq + hkv:])


@pytest.mark.parametrize("rows,experts", [(1, 16), (2, 3), (4, 16), (5, 20), (8, 16), (9, 40), (13, 7), (16, 128), (17, 130), (28, 33), (32, 256), (33, 9)])
@pytest.mark.parametrize("H", [256, 768, 4096])
def test_router_projection(fab, H, rows, experts):  # noqa: F811
    """Every row and expert remainder of a tile's register blocks, from global memory and (9 to 32 rows) through the ring, bit for
    bit."""
    import oracle
    g = torch.Generator().manual_seed(rows)
    x, wr = (torch.randn(n, H, generator=g).to(torch.bfloat16) for n in (rows, experts))
    xd, wd, out = x.cuda(), wr.cuda(), torch.zeros(rows, experts, device="cuda")
    args = torch.frombuffer(bytearray(pack("LogitsArgs", x=xd, wr=wd, logits=out, T=rows, H=H, E=experts)), dtype=torch.uint8).cuda()
    p = Program()
    run_program(fab, p, p.stage([Tile(48, i=(0, rows, 0, 0), a=(args.data_ptr(),))]))
    want = oracle.router_logits(oracle.bf16_bits(x), oracle.bf16_bits(wr))
    assert np.array_equal(out.cpu().numpy().view(np.int32), want.view(np.int32))


@pytest.mark.parametrize("divide,silu", [(0, 1), (1, 0)])
@pytest.mark.parametrize("e", [132, 256, 512, 516])
def test_head_norm_ahead_or_not(fab, e, divide, silu):  # noqa: F811
    """Tiles of more than four items load one item ahead (heads of 129 to 512 columns); tiles of four do not: the same bits."""
    g = torch.Generator(device="cuda").manual_seed(e)
    rows, heads = 13, 3
    oe = (e + (4 if divide else 3)) & ~3
    o, w = torch.randn(rows, heads, oe, generator=g, device="cuda"), torch.randn(heads, e, generator=g, device="cuda")
    if divide:
        o[:, :, e] = 0.5 + torch.rand(rows, heads, generator=g, device="cuda")
    gate = torch.randn(rows, heads * e, generator=g, device="cuda").to(torch.bfloat16)
    outs = []
    for per in (4, 5, rows * heads):
        out = torch.zeros(rows, heads * e, device="cuda", dtype=torch.bfloat16)
        block = pack("HeadNormArgs", o=o, g=gate, w=w, out=out, heads=heads, e=e, ld_g=heads * e, ld_out=heads * e, eps=EPS, divide=divide, silu=silu,
                     w_head=e)
        torch.cuda.synchronize()
        run_rows(fab, 58, block, rows * heads, per)
        outs.append(out)
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    x = o[:, :, :e].double() / (o[:, :, e:e + 1].double() if divide else 1)
    z = gate.double().view(rows, heads, e)
    close(outs[0].view(rows, heads, e), over_rms(x) * w.double() * z.sigmoid() * (z if silu else 1), "out")


@pytest.mark.parametrize("embedding", [False, True])
@pytest.mark.parametrize("H", [256, 768, 2048, 2304])
def test_norm_rows_ahead_or_not(fab, H, embedding):  # noqa: F811
    """Tiles of eight rows and more load a row ahead (up to 2048 columns); tiles of four do not: the same bits."""
    g = torch.Generator(device="cuda").manual_seed(H)
    rows = 61
    table, w = (torch.randn(n, H, generator=g, device="cuda").to(torch.bfloat16) for n in (40, 1))
    tokens = torch.randint(0, 40, (rows,), generator=g, device="cuda", dtype=torch.int32)
    gather = torch.full((rows,), -1, dtype=torch.int32, device="cuda")
    gather[rows - 1], gather[1] = 0, 1
    outs = []
    for per in (4, 9, 28):
        x = torch.zeros(rows, H, device="cuda", dtype=torch.bfloat16) if embedding else table[tokens.long()]
        out, out2 = (torch.zeros(n, H, device="cuda", dtype=torch.bfloat16) for n in (rows, 2))
        more = dict(embed=table, tokens=tokens) if embedding else dict(gather=gather, out2=out2)
        block = pack("NormArgs", x=x, w=w, out=out, H=H, ld=H, eps=EPS, **more)
        torch.cuda.synchronize()
        run_rows(fab, 42 if embedding else 36, block, rows, per)
        outs.append((x, out, out2))
    for other in outs[1:]:
        for a, b in zip(outs[0], other):
            assert torch.equal(a, b)
    x, out, out2 = outs[0]
    assert torch.equal(x, table[tokens.long()])
    close(out, over_rms(x.double()) * w.double(), "out")
    assert embedding or torch.equal(out2, out[[rows - 1, 1]])
