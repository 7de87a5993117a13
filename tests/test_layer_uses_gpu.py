"""The layer entry the way programs use it: stored and decomposed heads in training at every width, a graph walked twice,
checkpointing, saved tensors that leave the GPU, a stream of its own."""
from types import SimpleNamespace

import pytest
import torch
from torch.utils.checkpoint import checkpoint

from oracle import saf_oracle as O
from tests.test_attn_layer_gpu import build
from tests.util import make_decomp, make_pattern

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,hd,B,T", [(4, 64, 2, 320), (4, 96, 1, 200), (3, 128, 2, 129)])
@pytest.mark.parametrize("pattern", ["dense", "decomposed", "both"])
def test_training_with_stored_and_decomposed_heads(H, hd, B, T, pattern):
    """Against the fp32 oracle's autograd; the gates are those of test_attn_layer_gpu (same chain of bf16 roundings, the
    stored pattern one more of them)."""
    from saf_b200.attention import SafCausalSelfAttention, rope_tables
    C, S = H * hd, (T + 63) // 64 * 64
    cfg = SimpleNamespace(n_embd=C, n_head=H, block_size=S, bias=False, dropout=0.0, position_encoding="rope",
                          rand_attn_prior_repr="dense" if pattern == "dense" else "decomposed", freeze_pattern_dtype="bfloat16")
    g = torch.Generator().manual_seed(T)
    m = SafCausalSelfAttention(cfg)
    ps = [m.q_proj.weight, m.k_proj.weight, m.v_proj.weight, m.c_proj.weight]
    with torch.no_grad():
        for p in ps:
            p.copy_((torch.randn(C, C, generator=g) * C ** -0.5).bfloat16())
    m = m.cuda().train()
    states, patt = [0] * H, torch.zeros(H, T, T)
    alpha, rho, z = make_decomp(H, T, seed=2, scale=0.5)
    if pattern != "decomposed":
        states[1], patt[1] = 1, make_pattern(1, T, seed=3)[0]
        m.freeze_heads([1], patt[1:2])
    if pattern != "dense":
        states[2] = 2
        m.freeze_heads_decomposed([2], alpha[2:3].cuda(), rho[2:3].cuda())
    cos, sin = rope_tables(hd, T, device="cuda")
    x = torch.randn(B, T, C, generator=g).bfloat16()
    w = torch.randn(B, T, C, generator=g).bfloat16()
    xd = x.float().cuda().requires_grad_(True)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        y = m(xd, rope=(cos.view(1, 1, T, hd), sin.view(1, 1, T, hd)))
    got = torch.autograd.grad(y, [xd, *ps], w.cuda())
    leaves = [x.float().requires_grad_(True), *[p.detach().float().cpu().requires_grad_(True) for p in ps]]
    ref = O.attention_layer(*leaves, states, patt, H, rope=O.rope_cache(hd, T), alpha=alpha, rho=rho, z=z)
    want = torch.autograd.grad(ref, leaves, w.float())
    assert O.rel_l2(y.float().cpu(), ref.detach()) <= 1.5e-2
    for name, a, b in zip(("dx", "dWq", "dWk", "dWv", "dWo"), got, want):
        assert O.rel_l2(a.float().cpu(), b) <= 3.5e-2, name
    for h in (h for h in range(H) if states[h]):
        for gw in got[1:3]:
            assert gw[h * hd:(h + 1) * hd].abs().max().item() == 0.0


def one_pass(m, x, rope, dy, run=None):
    x = x.detach().clone().requires_grad_(True)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        y = (run or (lambda t: m(t, rope=rope)))(x)
    return [y.detach().clone(), *torch.autograd.grad(y, [x, *m.parameters()], dy)]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_the_same_gradients_whichever_way_the_graph_is_kept(dtype):
    m, rope, _, g = build(4, 64, 333, [1], 8, dtype)
    x = torch.randn(2, 333, 256, generator=g).cuda().to(dtype)
    dy = torch.randn(2, 333, 256, generator=g).cuda().bfloat16()
    plain = one_pass(m, x, rope, dy)
    x2 = x.clone().requires_grad_(True)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        y = m(x2, rope=rope)
    first = torch.autograd.grad(y, [x2, *m.parameters()], dy, retain_graph=True)
    m(torch.randn_like(x), rope=rope) if dtype == torch.bfloat16 else None      # another pass in between
    again = torch.autograd.grad(y, [x2, *m.parameters()], dy)
    again_from_file = one_pass(m, x, rope, dy, lambda t: checkpoint(lambda u: m(u, rope=rope), t, use_reentrant=False))
    with torch.autograd.graph.save_on_cpu():
        moved = one_pass(m, x, rope, dy)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        aside = one_pass(m, x, rope, dy)
    torch.cuda.current_stream().wait_stream(s)
    for other in ([plain[0], *first], [plain[0], *again], again_from_file, moved, aside):
        for a, b in zip(plain, other):
            assert torch.equal(a, b)


def test_checkpointed_fp32_layer():
    """The operators' own backward, which an fp32 layer walks."""
    m, rope, _, g = build(4, 64, 200, [1], 9, torch.float32)
    x = torch.randn(1, 200, 256, generator=g).cuda()
    dy = torch.randn(1, 200, 256, generator=g).cuda()
    got = []
    for run in (lambda t: m(t, rope=rope), lambda t: checkpoint(lambda u: m(u, rope=rope), t, use_reentrant=False)):
        xx = x.clone().requires_grad_(True)
        got.append(torch.autograd.grad(run(xx), [xx, *m.parameters()], dy))
    for a, b in zip(*got):
        assert torch.equal(a, b)


def test_inference_and_training_captured_into_graphs():
    """Replays follow the inputs and weights in place, as eager calls do."""
    from saf_b200.block import SafBlock
    m, rope, _, g = build(4, 64, 300, [2], 4, torch.float32)
    cfg = SimpleNamespace(n_embd=256, n_head=4, block_size=300, bias=False, dropout=0.0, position_encoding="rope")
    b = SafBlock(cfg)
    b.main_block.freeze_heads_sink_decay([1], [0.2], [0.9])
    b = b.cuda().bfloat16().eval()
    x = torch.randn(2, 300, 256, generator=g).cuda().requires_grad_(True)
    xb = x.detach().bfloat16()
    dy = torch.randn(2, 300, 256, generator=g).cuda().bfloat16()

    def infer():
        with torch.inference_mode(False), torch.no_grad():
            return [b(b(xb, rope=rope), rope=rope)]

    def train():
        with torch.autocast("cuda", dtype=torch.bfloat16):
            y = m(x, rope=rope)
        return [y.detach(), *torch.autograd.grad(y, [x, *m.parameters()], dy)]

    for fn in (infer, train):
        s = torch.cuda.Stream()
        s.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(s):
            fn()
        torch.cuda.current_stream().wait_stream(s)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            static = fn()
        for _ in range(3):
            with torch.no_grad():
                x.copy_(torch.randn(x.shape, generator=g))
                xb.copy_(x)
                m.q_proj.weight.mul_(1.25)
                b.mlp.c_fc.weight.mul_(0.75)
                b.main_block.c_proj.weight.mul_(1.25)
            graph.replay()
            graph.replay()
            got = [t.clone() for t in static]
            for u, v in zip(got, fn()):
                assert torch.equal(u, v)


def test_two_threads_with_streams_of_their_own():
    import threading
    m, rope, _, g = build(4, 64, 500, [1], 12, torch.float32)
    xs = [torch.randn(2, 500, 256, generator=g).cuda() for _ in range(2)]
    dy = torch.randn(2, 500, 256, generator=g).cuda().bfloat16()
    want = [one_pass(m, x, rope, dy) for x in xs]
    torch.cuda.synchronize()
    bad = []

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(10):
                got = one_pass(m, xs[i], rope, dy)
                bad.extend(k for k, (a, b) in enumerate(zip(got, want[i])) if not torch.equal(a, b))
        torch.cuda.synchronize()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


@pytest.mark.parametrize("what", ["layer", "block", "backward"])
def test_the_first_cuda_call_of_a_thread(what):
    """Nothing on the thread has given it a context: the allocator serves from its cache and no torch kernel runs before."""
    import subprocess
    import sys
    import os
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    code = """
import sys, threading
sys.path[:0] = [%r, %r]
import torch
from types import SimpleNamespace
from saf_b200.block import SafBlock
torch.manual_seed(0)
b = SafBlock(SimpleNamespace(n_embd=256, n_head=4, block_size=64, bias=False, dropout=0.0, position_encoding="none"))
b = b.cuda().bfloat16().eval()
m, x = b.main_block, torch.randn(2, 64, 256).cuda().bfloat16().requires_grad_(True)
dy = torch.randn(2, 64, 256).cuda().bfloat16()
keep = []
def once():
    if %r == "backward":
        y = m(x)
        torch.empty(1 << 26, dtype=torch.uint8, device="cuda")       # what the backward allocates comes from this block
        torch.cuda.synchronize()
        keep.append(torch.autograd.grad(y, [x, *m.parameters()], dy)[0])
    else:
        with torch.inference_mode():
            keep.append(b(x) if %r == "block" else m(x))
if %r == "backward":
    once()                                                           # the engine's thread, on its first call
else:
    once(); once()
    keep.pop()                                                       # its output and workspace are free again
    torch.cuda.synchronize()
    t = threading.Thread(target=once); t.start(); t.join()
    assert len(keep) == 2 and torch.equal(keep[0], keep[1])
assert torch.isfinite(keep[-1].float()).all()
""" % (root, os.path.join(root, "selective-attention-freezing_b200"), what, what, what)
    subprocess.run([sys.executable, "-c", code], check=True, timeout=180)
