"""Dense FP8 GeGLU MLP and the feed-forward pre/post steps against the CPU oracle.
Bit-exact where both sides see the same bytes (norm outputs, FP8 codes, row scales,
finalize); 2e-2 relative L2 for the FP8 GEMM outputs."""
import ctypes

import numpy as np
import pytest
import torch

from tests import hashgen
from tests.oracle_api import EXPERTS, HIDDEN, TOP_K, DenseOracle, bf16_to_f32

pytestmark = pytest.mark.gpu
DENSE = 2112


def bits(t):
    return t.detach().contiguous().view(torch.int16).cpu().numpy().view(np.uint16)


def rel_l2(got, want):
    got, want = got.astype(np.float64), want.astype(np.float64)
    return float(np.linalg.norm(got - want) / max(np.linalg.norm(want), 1e-30))


def norm_weight(seed, device):
    return (1.0 + 0.25 * hashgen.hash_uniform(HIDDEN, seed, device)).to(torch.bfloat16)


@pytest.fixture(scope="module")
def dense_oracle(oracle):
    return DenseOracle(oracle)


@pytest.mark.parametrize("rows", [1, 5, 300])
def test_ff_prepare_bit_exact(dense_oracle, cuda_device, rows):
    from gevva_b200 import feedforward as ff
    x = hashgen.activations(rows, HIDDEN, 71, cuda_device)
    dw, ew, rs = norm_weight(1, cuda_device), norm_weight(2, cuda_device), norm_weight(3, cuda_device)
    got = ff.ff_prepare(x, dw, ew, rs)
    want = dense_oracle.ff_prepare(bits(x), bits(dw), bits(ew), bits(rs))
    for g, w, name in zip(got, want, ("dense", "expert", "router")):
        assert (bits(g) == w).all(), name


@pytest.mark.parametrize("rows", [444, 445, 888, 889, 1500])
def test_ff_prepare_row_after_row(dense_oracle, cuda_device, rows):
    """From 445 rows on a CTA takes row after row: one, two and more rows a CTA, whole and ragged."""
    test_ff_prepare_bit_exact(dense_oracle, cuda_device, rows)


def test_pack_fp8_matches_oracle(dense_oracle, cuda_device):
    from gevva_b200 import feedforward as ff
    w = hashgen.expert_weights_chunk(0, 1, 256, HIDDEN, 33, cuda_device)[0]
    q, scale = ff.pack_fp8(w)
    oq, oscale = dense_oracle.pack_fp8(w.cpu().numpy())
    assert scale == oscale and (q.cpu().numpy() == oq).all()


@pytest.fixture(scope="module")
def dense_weights(cuda_device):
    from gevva_b200 import feedforward as ff
    gate = hashgen.expert_weights_chunk(0, 1, DENSE, HIDDEN, 51, cuda_device)[0]
    up = hashgen.expert_weights_chunk(0, 1, DENSE, HIDDEN, 52, cuda_device)[0]
    down = hashgen.expert_weights_chunk(0, 1, HIDDEN, DENSE, 53, cuda_device)[0]
    gq, gs = ff.pack_fp8(gate)
    uq, us = ff.pack_fp8(up)
    dq, ds = ff.pack_fp8(down)
    return torch.cat([gq, uq]).contiguous(), dq, gs, us, ds


@pytest.mark.parametrize("tokens", [1, 37, 300])
def test_dense_mlp_stages(dense_oracle, dense_weights, cuda_device, tokens):
    from gevva_b200 import feedforward as ff
    gate_up, down, gs, us, ds = dense_weights
    mlp = ff.DenseMlp(gate_up, down, gs, us, ds, 512)
    x = hashgen.activations(tokens, HIDDEN, 81, cuda_device)
    out, out_scales = mlp.launch(x)
    torch.cuda.synchronize()
    # stage 1: row quantisation, bit-exact
    q, s = dense_oracle.quantize_rows(bits(x))
    assert (mlp.buffer(0, torch.uint8)[: tokens * HIDDEN].cpu().numpy().reshape(tokens, HIDDEN) == q).all()
    assert (mlp.buffer(1, torch.float32)[:tokens].cpu().numpy() == s).all()
    # stage 2: gate|up GEMM on the same FP8 bytes
    want_gu = dense_oracle.gemm(q, gate_up.cpu().numpy())
    got_gu = bits(mlp.buffer(2, torch.bfloat16)[: tokens * 2 * DENSE]).reshape(tokens, 2 * DENSE)
    assert rel_l2(bf16_to_f32(got_gu), bf16_to_f32(want_gu)) < 5e-3
    # stage 3: GeGLU + requantise, bit-exact given the GPU's own gate|up output
    pq, ps = dense_oracle.gelu_quantize(got_gu, s, gs, us)
    assert (mlp.buffer(3, torch.uint8)[: tokens * DENSE].cpu().numpy().reshape(tokens, DENSE) == pq).all()
    assert (out_scales.cpu().numpy() == ps).all()
    # stage 4: down GEMM
    want_out = dense_oracle.gemm(pq, down.cpu().numpy())
    assert rel_l2(bf16_to_f32(bits(out)), bf16_to_f32(want_out)) < 5e-3


@pytest.mark.parametrize("tokens", [2, 3])
def test_dense_mlp_of_a_few_rows(dense_oracle, dense_weights, cuda_device, tokens):
    """The two launches of up to two tokens (one token above), and the first size beyond."""
    test_dense_mlp_stages(dense_oracle, dense_weights, cuda_device, tokens)


@pytest.mark.parametrize("tokens", [512, 513, 897, 1025])
def test_dense_mlp_rows_do_not_depend_on_the_batch(dense_weights, cuda_device, tokens):
    """Batches of several row tiles give every row the bits it has in a batch of 100, which is one tile."""
    from gevva_b200 import feedforward as ff
    gate_up, down, gs, us, ds = dense_weights
    mlp = ff.DenseMlp(gate_up, down, gs, us, ds, tokens)
    x = hashgen.activations(tokens, HIDDEN, 82, cuda_device)
    out, scales = (t.clone() for t in mlp.launch(x))
    hidden = mlp.buffer(2, torch.bfloat16)[: tokens * 2 * DENSE].view(tokens, -1).clone()
    for first in range(0, tokens, 100):
        rows = min(100, tokens - first)
        part, part_scales = mlp.launch(x[first : first + rows].contiguous())
        assert torch.equal(mlp.buffer(2, torch.bfloat16)[: rows * 2 * DENSE].view(rows, -1), hidden[first : first + rows])
        assert torch.equal(part[:rows], out[first : first + rows])
        assert torch.equal(part_scales[:rows], scales[first : first + rows])
    assert out.float().abs().max() > 0


@pytest.mark.parametrize("tokens", [1, 2])
@pytest.mark.parametrize("of", [3, 100])
def test_dense_mlp_of_a_few_rows_has_the_bits_of_a_larger_batch(dense_weights, cuda_device, tokens, of):
    """One and two tokens have launches of their own (dense_few_rows.cu): every row of theirs, codes, scales, unscaled projections and all, has
    the bits that it has in a batch of three or of a hundred."""
    from gevva_b200 import feedforward as ff
    gate_up, down, gs, us, ds = dense_weights
    mlp = ff.DenseMlp(gate_up, down, gs, us, ds, of)

    def launch(x):
        rows = len(x)
        out, _ = mlp.launch(x.contiguous())
        parts = [mlp.buffer(i, dtype)[: rows * width].view(rows, width)
                 for i, dtype, width in ((0, torch.uint8, HIDDEN), (1, torch.float32, 1), (2, torch.bfloat16, 2 * DENSE),
                                         (3, torch.uint8, DENSE), (4, torch.float32, 1))] + [out]
        return [part.clone().view(torch.uint8) for part in parts]

    x = hashgen.activations(of, HIDDEN, 84, cuda_device)
    x[1] *= 4096.0
    x[2] = 0.0
    whole = launch(x)
    for first in range(0, of - tokens + 1):
        for got, want in zip(launch(x[first : first + tokens]), whole):
            assert torch.equal(got, want[first : first + tokens]), first
    mlp.check()


@pytest.mark.parametrize("tokens", [1, 2])
@pytest.mark.parametrize("concurrent", [False, True])
def test_layers_of_a_few_tokens_have_the_bits_of_a_larger_batch(cuda_device, tokens, concurrent):
    """A token decoded alone and the same one among forty, through four whole layers."""
    from gevva_b200.synthetic import SyntheticStack
    stack = SyntheticStack(4, 40, cuda_device, seed=12)
    hidden = hashgen.activations(40, HIDDEN, 85, cuda_device)
    want = stack.forward(hidden, concurrent=False).clone()
    for first in range(0, 40, 4):
        assert torch.equal(stack.forward(hidden[first : first + tokens].contiguous(), concurrent=concurrent), want[first : first + tokens]), first
    for layer in stack.layers:
        layer.experts.check()


def test_ff_finalize_bit_exact(dense_oracle, cuda_device):
    from gevva_b200 import feedforward as ff
    rows = 41
    dense = hashgen.activations(rows, HIDDEN, 91, cuda_device)
    routes = hashgen.activations(rows * TOP_K, HIDDEN, 92, cuda_device)
    residual = hashgen.activations(rows, HIDDEN, 93, cuda_device)
    gen = torch.Generator().manual_seed(4)
    rw = (torch.rand((rows, TOP_K), generator=gen) * 0.3).to(cuda_device)
    inverse = torch.randperm(rows * TOP_K, generator=gen).to(torch.int32).to(cuda_device)
    act_scales = (0.5 + torch.rand(rows, generator=gen)).to(cuda_device)
    dw, ew, cw = norm_weight(4, cuda_device), norm_weight(5, cuda_device), norm_weight(6, cuda_device)
    scalar = torch.tensor([0.75], dtype=torch.bfloat16, device=cuda_device)
    for scales, proj in ((act_scales, 0.013), (None, 1.0)):
        proj_dev = None if scales is None else torch.tensor([proj], dtype=torch.float32, device=cuda_device)
        got = ff.ff_finalize(dense, dw, routes, rw, inverse, ew, cw, residual, scalar, scales, proj_dev)
        want = dense_oracle.finalize(bits(dense), bits(dw), bits(routes), rw.cpu().numpy(),
                                     inverse.cpu().numpy(), bits(ew), bits(cw), bits(residual),
                                     bits(scalar)[0], None if scales is None else scales.cpu().numpy(), float(np.float32(proj)))
        assert (bits(got) == want).all()


def test_layer_wiring_against_oracle(oracle, dense_oracle, dense_weights, cuda_device):
    """One layer of the FFN stack (pre-norms, router, experts beside the dense MLP, fused
    finalize) against the same chain on the CPU; the router logits are shared so that both
    sides route identically."""
    import gevva_b200 as gm
    from gevva_b200 import feedforward as ff
    from gevva_b200.synthetic import make_packed_experts
    tokens = 24
    p = make_packed_experts(3, cuda_device, chunk=32)
    s1, s2 = 6.0 / 2688.0, 8.0 / 2688.0
    ones = torch.ones(EXPERTS, dtype=torch.float32, device=cuda_device)
    w = gm.ExpertWeights(p["w13"], p["w13_sf"], p["w2"], p["w2_sf"], (p["g13"] * s1).contiguous(),
                         (p["g2"] * s2).contiguous(), (ones / s1).contiguous(), (ones / s2).contiguous())
    gate_up, down, gs, us, ds = dense_weights
    dw, ew, rs = norm_weight(1, cuda_device), norm_weight(2, cuda_device), norm_weight(3, cuda_device)
    dpost, epost, cpost = norm_weight(4, cuda_device), norm_weight(5, cuda_device), norm_weight(6, cuda_device)
    scalar = torch.tensor([0.5], dtype=torch.bfloat16, device=cuda_device)
    router_w = (hashgen.hash_uniform(EXPERTS * HIDDEN, 5, cuda_device) * 0.0346).view(EXPERTS, HIDDEN).to(
        torch.bfloat16)
    layer = ff.FeedForwardLayer(dw, ew, rs, router_w, torch.ones(EXPERTS, dtype=torch.bfloat16, device=cuda_device),
                                dpost, epost, cpost, scalar, gm.Nvfp4ExpertRunner(w, 64),
                                ff.DenseMlp(gate_up, down, gs, us, ds, 64))
    hidden = hashgen.activations(tokens, HIDDEN, 101, cuda_device)
    got = layer.forward(hidden, torch.cuda.Stream(device=cuda_device))
    torch.cuda.synchronize()
    # CPU chain
    dense_in, expert_in, router_in = dense_oracle.ff_prepare(bits(hidden), bits(dw), bits(ew), bits(rs))
    # the library's own logits (fused projection, deterministic), so that both sides route alike
    _, _, logits = gm.route_project(torch.from_numpy(router_in.view(np.int16)).to(cuda_device).view(torch.bfloat16),
                                    router_w, torch.ones(EXPERTS, dtype=torch.bfloat16, device=cuda_device),
                                    want_logits=True)
    rw, ids = oracle.route(bits(logits), bits(torch.ones(EXPERTS, dtype=torch.bfloat16)))
    hw = dict(w13=p["w13"].cpu().numpy(), w13_sf=p["w13_sf"].cpu().numpy(), w2=p["w2"].cpu().numpy(),
              w2_sf=p["w2_sf"].cpu().numpy(), alpha1=w.alpha1.cpu().numpy(), alpha2=w.alpha2.cpu().numpy(),
              in_scale_q1=w.in_scale_q1.cpu().numpy(), in_scale_q2=w.in_scale_q2.cpu().numpy())
    _, routed, inverse = oracle.moe_layer(expert_in, ids, rw, hw, want_routed=True)
    q, s = dense_oracle.quantize_rows(dense_in)
    pq, ps = dense_oracle.gelu_quantize(dense_oracle.gemm(q, gate_up.cpu().numpy()), s, gs, us)
    dense_out = dense_oracle.gemm(pq, down.cpu().numpy())
    want = dense_oracle.finalize(dense_out, bits(dpost), routed, rw, inverse, bits(epost), bits(cpost),
                                 bits(hidden), bits(scalar)[0], ps, ds)
    assert rel_l2(bf16_to_f32(bits(got)), bf16_to_f32(want)) < 2e-2


def test_ffn_stack_runs_at_configured_size(cuda_device):
    """30 layers x 2048 tokens: finite output, identical on a second pass, and the two-stream
    schedule equals the single-stream one."""
    from gevva_b200.synthetic import SyntheticStack
    stack = SyntheticStack(30, 2048, cuda_device, distinct_experts=False)
    hidden = hashgen.activations(2048, HIDDEN, 7, cuda_device)
    a = stack.forward(hidden)
    b = stack.forward(hidden)
    c = stack.forward(hidden, concurrent=False)
    torch.cuda.synchronize()
    assert torch.isfinite(a.float()).all() and a.float().abs().max() > 0
    assert torch.equal(a, b) and torch.equal(a, c)


def test_thirty_layers_captured_into_one_graph_at_verifier_size(cuda_device):
    """The decode-side caller of the path: rows = sessions x (drafts + 1) <= 40, the whole
    30-layer enqueue (prepare -> router -> route -> experts unreduced beside the dense MLP on a
    second stream -> finalize) captured once and replayed (src/cuda/runtime/verifier.cuh:960-1042,
    capture :1058-1078).  Replays must reproduce the eager pass bit for bit, also after the input
    buffer has been refilled."""
    from gevva_b200.synthetic import SyntheticStack
    rows = 40
    stack = SyntheticStack(30, rows, cuda_device, distinct_experts=False)
    first = hashgen.activations(rows, HIDDEN, 11, cuda_device)
    second = hashgen.activations(rows, HIDDEN, 12, cuda_device)
    want_first = stack.forward(first, concurrent=False).clone()
    want_second = stack.forward(second, concurrent=False).clone()
    torch.cuda.synchronize()
    assert not torch.equal(want_first, want_second)
    static_in = first.clone()
    stack.forward(static_in)            # warm-up outside the capture
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        static_out = stack.forward(static_in)
    for _ in range(2):
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(static_out, want_first)
    static_in.copy_(second)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(static_out, want_second)
    for layer in stack.layers:
        layer.experts.check()


@pytest.mark.parametrize("tokens", [1, 2, 16, 128, 129, 301])
def test_layer_call_equals_its_parts(cuda_device, tokens):
    """gevva_ff_layer_launch against the calls it stands for, made one by one: the same bits, on one
    stream and with the dense MLP on a second one, where the two sides share the SMs."""
    from gevva_b200 import feedforward as ff
    from gevva_b200.runtime import route_project
    from gevva_b200.synthetic import SyntheticStack
    stack = SyntheticStack(1, 512, cuda_device, seed=5)
    layer = stack.layers[0]
    hidden = hashgen.activations(tokens, HIDDEN, 21 + tokens, cuda_device)
    dense_in, expert_in, router_in = ff.ff_prepare(hidden, layer.dense_pre, layer.expert_pre, layer.router_scale)
    weights, ids = route_project(router_in, layer.router_w, layer.expert_scale, status_of=layer.experts)
    dense_out, dense_scales = layer.dense.launch(dense_in)
    layer.experts.launch_batch_unreduced(expert_in, ids, tokens)
    want = ff.ff_finalize(dense_out, layer.dense_post, layer.experts.routed_output(), weights,
                          layer.experts.inverse_routes(), layer.expert_post, layer.combined_post, hidden,
                          layer.layer_scalar, dense_scales, layer.dense.projection_scale)
    for aux in (None, torch.cuda.Stream(device=cuda_device)):
        for _ in range(2):
            got = layer.forward(hidden, aux)
        torch.cuda.synchronize()
        assert torch.equal(got, want)
    layer.experts.check()


@pytest.mark.parametrize("tokens,widths", [(1, (128, 128)), (3, (128, 128)), (5, (128, 128)), (8, (256, 256)), (100, (256, 256)), (200, (256, 256)),
                                           (300, (256, 256)), (512, (128, 256)), (640, (256, 256))])
def test_dense_mlp_beside_the_experts(cuda_device, tokens, widths):
    """The one-CTA kernels that the dense MLP takes on its share of a layer's SMs, with 128 or 256 weight rows an item in either
    projection, against the pair kernels of the MLP alone: its input, its gate and up projection and its unscaled output.
    (One token: the kernels of dense_few_rows.cu in both places.)"""
    from gevva_b200 import feedforward as ff
    from gevva_b200.synthetic import SyntheticStack
    sms = next(share for last, share in ((4, 48), (6, 33), (12, 17), (128, 16), (256, 22), (640, 33)) if tokens <= last)
    tiles = (tokens + 127) // 128
    items = lambda n_out, width: -(-tiles * -(-n_out // width) // sms)
    assert widths == tuple(256 if 3 * items(n, 256) <= 2 * items(n, 128) else 128 for n in (2 * DENSE, HIDDEN))  # the library's rule
    layer = SyntheticStack(1, 640, cuda_device, seed=6).layers[0]
    lib = ff._lib()
    hidden = hashgen.activations(tokens, HIDDEN, 55 + tokens, cuda_device)
    out = torch.empty_like(hidden)
    workspace = torch.zeros(lib.gevva_ff_layer_workspace_bytes(tokens), dtype=torch.uint8, device=cuda_device)
    parts = ("dense_pre", "expert_pre", "router_scale", "router_w", "expert_scale", "dense_post", "expert_post", "combined_post",
             "layer_scalar")
    native = ff._Layer(*[getattr(layer, p).data_ptr() for p in parts], layer.experts._handle, layer.dense._handle)
    aux = torch.cuda.Stream(device=cuda_device)
    torch.cuda.synchronize()
    assert lib.gevva_ff_layer_launch(ctypes.byref(native), hidden.data_ptr(), out.data_ptr(), workspace.data_ptr(), tokens,
                                     torch.cuda.current_stream().cuda_stream, aux.cuda_stream) == 0
    torch.cuda.synchronize()
    layer.experts.check()
    rows = tokens * HIDDEN * 2  # a multiple of 256, so the workspace's four row buffers lie end to end
    dense_in = workspace[:rows].view(torch.bfloat16).view(tokens, HIDDEN)
    dense_out = workspace[3 * rows : 4 * rows].view(torch.bfloat16).view(tokens, HIDDEN)
    gate_up = layer.dense.buffer(2, torch.bfloat16)[: tokens * 2 * DENSE].clone()
    alone, _ = layer.dense.launch(dense_in)
    layer.dense.check()
    assert torch.equal(layer.dense.buffer(2, torch.bfloat16)[: tokens * 2 * DENSE], gate_up)
    assert torch.equal(alone, dense_out) and alone.float().abs().max() > 0


@pytest.mark.parametrize("tokens", [130, 256, 257, 296, 640, 641])
def test_layers_beside_the_dense_mlp_in_a_graph(cuda_device, tokens):
    """Layers of the sizes whose experts stream share the SMs with the dense MLP: a captured stack of three gives the bits of
    the same layers on one stream, at the edges of the table of shares and of the range."""
    from gevva_b200.synthetic import SyntheticStack
    stack = SyntheticStack(3, 641, cuda_device, seed=9, distinct_experts=False)
    hidden = hashgen.activations(tokens, HIDDEN, 5 + tokens, cuda_device)
    want = stack.forward(hidden, concurrent=False).clone()
    stack.forward(hidden)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = stack.forward(hidden)
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, want)
    for layer in stack.layers:
        layer.experts.check()


@pytest.mark.parametrize("tokens", [17, 127, 129, 255, 257, 1153, 2048])
def test_dense_pairs_at_tile_edges(dense_weights, cuda_device, tokens):
    """The dense GEMMs by CTA pairs take 256 tokens and 256 or 192 columns an item and store 16 rows a step: whole and ragged last
    tiles, with either width, give every row the bits it has in a batch of 112 (one ragged tile), and store nothing past the end."""
    from gevva_b200 import feedforward as ff
    gate_up, down, gs, us, ds = dense_weights
    mlp = ff.DenseMlp(gate_up, down, gs, us, ds, tokens + 300)
    x = hashgen.activations(tokens, HIDDEN, 83, cuda_device)
    guarded = torch.full((tokens + 256, HIDDEN), 7.0, device=cuda_device, dtype=torch.bfloat16)
    mlp.buffer(2, torch.bfloat16).fill_(5.0)
    mlp.launch(x, out=guarded[:tokens])
    hidden = mlp.buffer(2, torch.bfloat16).view(-1, 2 * DENSE).clone()
    assert (guarded[tokens:] == 7.0).all() and (hidden[tokens:] == 5.0).all()
    for first in range(0, tokens, 112):
        rows = min(112, tokens - first)
        part, _ = mlp.launch(x[first : first + rows].contiguous())
        assert torch.equal(mlp.buffer(2, torch.bfloat16)[: rows * 2 * DENSE].view(rows, -1), hidden[first : first + rows])
        assert torch.equal(part[:rows], guarded[first : first + rows])
    assert guarded[:tokens].float().abs().max() > 0


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("tokens", [1, 3, 600, 2048])
def test_weights_written_right_before_the_dense_mlp(dense_weights, cuda_device, tokens, graph):
    """The dense GEMMs fetch weights before the kernel in front of them has ended.  What kernels in front of the whole call write is there all
    the same, also where those let their successors start before they have written anything: ff_prepare, whose normalised rows of
    ones are its norm weight, whose bytes are the MLP's weights here.  The last hundred rows that it writes come behind a w2 on four
    SMs, which takes a millisecond and lets it start at its own beginning, so a call that did not wait for it would find what was there before.
    For the MLP by itself and for a layer's, on the same stream and on a second one."""
    from gevva_b200 import feedforward as ff
    from gevva_b200.runtime import STAGE_W2
    from gevva_b200.synthetic import SyntheticStack
    gate_up, down, gs, us, ds = dense_weights
    lib = ff._lib()
    ones = torch.ones((DENSE, HIDDEN), dtype=torch.bfloat16, device=cuda_device)
    unused = [torch.empty_like(ones) for _ in range(2)]
    stack = SyntheticStack(1, 2600, cuda_device, seed=11)
    delay = stack.layers[0].experts
    stack.forward(hashgen.activations(2600, HIDDEN, 94, cuda_device))  # (a plan and operands for the w2)
    launch_on = lib["_ZN2gv20moe_launch_stages_onEP9gevva_moePKvPKiPKfPvijP11CUstream_sti"]  # gv::moe_launch_stages_on
    launch_on.argtypes = [ctypes.c_void_p] * 5 + [ctypes.c_int, ctypes.c_uint, ctypes.c_void_p, ctypes.c_int]
    generator = torch.Generator(device=cuda_device).manual_seed(tokens)
    # two rows of bf16 values, both of whose bytes are finite E4M3 numbers: 0.5 to 2 in steps of 1/256 and up, of either sign
    rows = [(torch.randint(0x3F00, 0x3F7F, (HIDDEN,), generator=generator, device=cuda_device) +
             0x8000 * torch.randint(0, 2, (HIDDEN,), generator=generator, device=cuda_device)).to(torch.uint16).view(torch.bfloat16)
            for _ in range(2)]

    def write(weights, row, count=DENSE):
        stream = torch.cuda.current_stream().cuda_stream
        for buffer in weights:
            assert lib.gevva_ff_prepare(ones.data_ptr(), row.data_ptr(), row.data_ptr(), row.data_ptr(), buffer.data_ptr(), unused[0].data_ptr(),
                                        unused[1].data_ptr(), min(count, buffer.numel() // (2 * HIDDEN)), stream) == 0

    def check(weights, run):
        want, calls = [], []
        for row, other in zip(rows, reversed(rows)):
            write(weights, row)
            torch.cuda.synchronize()
            assert all(torch.equal(buffer.view(torch.bfloat16).view(-1, HIDDEN), row.expand(buffer.numel() // (2 * HIDDEN), HIDDEN))
                       for buffer in weights)
            want.append(run().clone())
            torch.cuda.synchronize()

            def call(row=row, other=other):
                write(weights, row)
                write(weights[:1], other, 100)
                assert launch_on(delay._handle, None, None, None, None, 2600, STAGE_W2, torch.cuda.current_stream().cuda_stream, 4) == 0
                write(weights[:1], row, 100)
                return run()

            if graph:
                captured = torch.cuda.CUDAGraph()
                with torch.cuda.graph(captured):
                    out = call()
                calls.append(lambda captured=captured, out=out: (captured.replay(), out)[1])
            else:
                calls.append(call)
        assert want[0].isfinite().all() and not torch.equal(*want)
        for turn in range(6):
            assert torch.equal(calls[turn % 2](), want[turn % 2])

    x = hashgen.activations(tokens, HIDDEN, 95, cuda_device)
    mlp = ff.DenseMlp(gate_up.clone(), down.clone(), gs, us, ds, tokens)
    check(mlp._keep, lambda: mlp.launch(x)[0])
    layer = SyntheticStack(1, max(tokens, 64), cuda_device, seed=12).layers[0]
    aux = torch.cuda.Stream(device=cuda_device)
    check(layer.dense._keep, lambda: layer.forward(x))
    check(layer.dense._keep, lambda: layer.forward(x, aux_stream=aux))
    delay.check()


@pytest.mark.parametrize("tokens", [1, 3, 129, 600])
def test_dense_output_aligned_to_16_bytes(dense_weights, cuda_device, tokens):
    """An output that starts between two 32-byte lines gets the bits of one that does not, and nothing around it."""
    from gevva_b200 import feedforward as ff
    gate_up, down, gs, us, ds = dense_weights
    mlp = ff.DenseMlp(gate_up, down, gs, us, ds, tokens)
    x = hashgen.activations(tokens, HIDDEN, 84, cuda_device)
    want = mlp.launch(x)[0].clone()
    flat = torch.full((tokens * HIDDEN + 16,), 7.0, device=cuda_device, dtype=torch.bfloat16)
    assert flat.data_ptr() % 32 == 0
    mlp.launch(x, out=flat[8:-8].view(tokens, HIDDEN))
    assert torch.equal(flat[8:-8].view(tokens, HIDDEN), want)
    assert (flat[:8] == 7.0).all() and (flat[-8:] == 7.0).all()


def test_dense_status_is_read_and_cleared(dense_weights, cuda_device):
    """The word that an expired wait of the dense kernels sets (here a store stands in for it) is what last_status() returns, once."""
    import gevva_b200 as gm
    from gevva_b200 import feedforward as ff
    from gevva_b200.runtime import _view
    mlp = ff.DenseMlp(*dense_weights, 300)
    mlp.launch(hashgen.activations(300, HIDDEN, 85, cuda_device))
    mlp.check()
    _view(ff._lib().gevva_dense_status_word(mlp._handle), (1,), torch.int32, cuda_device).fill_(2)
    with pytest.raises(gm.GevvaMoeError, match="wait expired"):
        mlp.check()
    assert mlp.last_status() == 0


@pytest.mark.parametrize("tokens,gate_scale", [(593, 1.0), (600, 1e-6), (1023, 1e6), (1024, 1e-5), (2369, 3e-6)])
def test_activation_of_large_batches_equals_the_small_ones(dense_weights, cuda_device, tokens, gate_scale):
    """From five tokens an SM the GELU step takes a warp a row and looks its tanh factor up, from 1024 tokens the first quantiser takes a
    warp a row: all bytes and scales as in batches of 64, for gates inside the table, past both of its ends, and zero."""
    from gevva_b200 import feedforward as ff
    gate_up, down, gs, us, ds = dense_weights
    mlp = ff.DenseMlp(gate_up, down, gs * gate_scale, us, ds, tokens)
    x = hashgen.activations(tokens, HIDDEN, 89, cuda_device)
    x[tokens // 2].zero_()
    views = lambda rows: (mlp.buffer(0, torch.uint8)[: rows * HIDDEN].view(rows, -1), mlp.buffer(1, torch.float32)[:rows],
                          mlp.buffer(3, torch.uint8)[: rows * DENSE].view(rows, -1), mlp.buffer(4, torch.float32)[:rows])
    mlp.launch(x)
    whole = [v.clone() for v in views(tokens)]
    for first in range(0, tokens, 64):
        rows = min(64, tokens - first)
        mlp.launch(x[first : first + rows].contiguous())
        for part, all_rows in zip(views(rows), whole):
            assert torch.equal(part, all_rows[first : first + rows])
    assert whole[2].count_nonzero() > 0
