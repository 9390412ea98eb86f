"""The matrix memory's tile (kind 57) on its own: four-token steps of 32 and 64 columns (a[1]) and one token at a time (a[1] = 0)
against the recurrence in 64 bits, at the edges of steps, of chunks of 32 tokens and of column blocks."""
import numpy as np
import pytest
import torch

from monoserve_b200.fabric import Program, Tile
from monoserve_b200.fabric.args import pack
from tests.test_gpu_fabric_gemm import fab, run_program  # noqa: F401

pytestmark = pytest.mark.gpu

K_MEMORY, HEADS, CAP = 57, 2, 15.0


class Portion:
    """`rows` tokens of one request at slot 1: bf16 projections, gates in two slabs, and where `past`, a state to go on from."""

    def __init__(self, d, e, rows, past, seed):
        g = torch.Generator(device="cuda").manual_seed(seed)
        r = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
        self.d, self.e, self.rows, self.past = d, e, rows, past
        self.ld = -(-HEADS * (2 * d + e) // 8) * 8
        self.proj = r(rows, self.ld).to(torch.bfloat16)
        self.gates, self.bias = 0.7 * r(2, rows + 3, 2 * HEADS), torch.cat([r(HEADS), 3 + r(HEADS)])
        dp, copies = (d + 3) & ~3, (e + 32) // 32
        self.state0, self.m0 = torch.zeros(2, HEADS, e + 1, dp, device="cuda"), torch.zeros(2, HEADS, copies, device="cuda")
        if past:
            self.state0[1, :, :, :d] = r(HEADS, e + 1, d)
            self.m0[1] = r(HEADS, 1)
        self.pos = torch.arange(past, past + rows, dtype=torch.int32, device="cuda")

    def run(self, fab, width):  # noqa: F811
        d, e, at = self.d, self.e, self.proj.data_ptr()
        oe = (e + 4) & ~3
        state, m, out = self.state0.clone(), self.m0.clone(), torch.zeros(self.rows, HEADS, oe, device="cuda")
        block = pack("MemoryArgs", q=at, k=at + 2 * HEADS * d, v=at + 4 * HEADS * d, gates=self.gates, gate_parts=2,
                     gate_rows=self.rows + 3, gate_bias=self.bias, state=state, m=m, out=out, tok_pos=self.pos, ld_qkv=self.ld,
                     ld_gates=2 * HEADS, heads=HEADS, d=d, e=e, f32=0, q_scale=d ** -0.5, cap=CAP)
        args = torch.frombuffer(bytearray(block), dtype=torch.uint8).cuda()
        torch.cuda.synchronize()
        p = Program()
        tiles = [Tile(K_MEMORY, i=(0, self.rows, h | c << 16, 1), a=(args.data_ptr(), width))
                 for h in range(HEADS) for c in range(-(-(e + 1) // (width or 32)))]
        run_program(fab, p, p.stage(tiles))
        assert torch.equal(state[0], self.state0[0]) and torch.equal(m[0], self.m0[0])   # another request's
        return out[:, :, :e + 1], state[1, :, :, :d], m[1]

    def exact(self):
        d, e, H = self.d, self.e, HEADS
        x = self.proj.double()
        q, k, v = (x[:, a:a + H * n].view(self.rows, H, n) for a, n in ((0, d), (H * d, d), (2 * H * d, e)))
        z = CAP * torch.tanh((self.gates[:, :self.rows].double().sum(0) + self.bias.double()) / CAP)
        i, f = z[:, :H], torch.nn.functional.logsigmoid(z[:, H:])
        v = torch.cat([v, v.new_ones(self.rows, H, 1)], -1)
        S, top, out = self.state0[1, :, :, :d].double(), self.m0[1, :, 0].double(), []
        for t in range(self.rows):
            new = torch.maximum(f[t] + top, i[t])
            S = (f[t] + top - new).exp()[:, None, None] * S + ((i[t] - new).exp()[:, None] * v[t])[..., None] * k[t][:, None]
            top = new
            o = torch.einsum("hed,hd->he", S, q[t] * d ** -0.5)
            o[:, e] = torch.maximum(o[:, e].abs(), (-top).exp()) + 1e-6
            out.append(o)
        return torch.stack(out), S, top[:, None].expand_as(self.m0[1])


def distance(got, want):
    return float((got.double() - want).norm() / want.norm())


# d: 128 and 256 with whole column blocks take the staging of whole chunks (rows in 16-byte pieces, none of them padding)
@pytest.mark.parametrize("past", [0, 5])
@pytest.mark.parametrize("rows", [2, 3, 31, 32, 33, 70])
@pytest.mark.parametrize("d,e", [(24, 40), (128, 64), (128, 95), (130, 31), (256, 63), (256, 512), (18, 1)])
def test_steps_of_four_tokens(fab, d, e, rows, past):  # noqa: F811
    """fp32 sums of up to 256 products and 70 tokens: 2^-24 of each term, and the gates' exponentials of sums of up to 70
    logarithms: about 1e-6 in all.  The steps are no further from 64 bits than one token at a time is, give or take a quarter."""
    p = Portion(d, e, rows, past, seed=d + e + rows)
    want = p.exact()
    single = [distance(a, b) for a, b in zip(p.run(fab, 0), want)]
    for width in (32, 64):
        for what, got, exact, one in zip(("out", "state", "m"), p.run(fab, width), want, single):
            err = distance(got, exact)
            assert err < 5e-6 and err < 1.25 * one + 2e-7, (width, what, err, one)


@pytest.mark.parametrize("width", [0, 32, 64])
@pytest.mark.parametrize("at", [4, 5, 6, 7, 34])
def test_a_token_is_not_reached_by_later_ones(fab, at, width):  # noqa: F811
    """Values that are not finite at one token leave the outputs of the tokens before it as they are, also inside a step."""
    p = Portion(128, 64, 40, 0, seed=at)
    clean = p.run(fab, width)[0]
    p.proj[at, 2 * HEADS * p.d:] = float("inf")
    p.proj[at, HEADS * p.d:HEADS * p.d + 3] = float("nan")
    got = p.run(fab, width)[0]
    assert torch.equal(got[:at], clean[:at]) and not bool(torch.isfinite(got[at]).all())
