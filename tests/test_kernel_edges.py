"""Small cases at the edges of the kernels' tiles, steps and dispatch rules, against the CPU oracle or bit for bit against
another route to the same result."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from oracle import quant  # noqa: E402
from test_cuda_moe import FULL, Layer, QT, check_layer, dev, make, padded_slab_layer, pkg  # noqa: E402,F401


@pytest.mark.parametrize("n,dims", [(16, dict(H=128, E=2, K=2, F=128, S=128)), (17, dict(H=256, E=3, K=1, F=128, S=384)),
                                    (191, dict(H=128, E=2, K=2, F=128, S=128)), (192, dict(H=128, E=2, K=2, F=256, S=128)),
                                    (193, dict(H=384, E=2, K=2, F=128, S=256)), (385, dict(H=128, E=4, K=2, F=128, S=128))])
def test_fp16_grouped_gemm_at_tile_edges(pkg, port, n, dims):
    """fp16 weights by TMA: K of two blocks up (fewer than the ring's stages), ragged token tiles, one to several weight tiles."""
    L, hidden, resid = make(300 + n, dims, "f16", n)
    check_layer(pkg, port, L, hidden, resid, gemm=True)


def test_fp16_grouped_gemm_honours_a_mixed_layer(pkg, port):
    """Quantised experts beside an fp16 shared MLP: both weight operands of the kernel in one call."""
    L, hidden, resid = make(41, dict(H=256, E=4, K=2, F=128, S=256), "q8_0", 70, shared_qname="f16")
    check_layer(pkg, port, L, hidden, resid, gemm=True)


@pytest.mark.parametrize("hot", ["gate", "up", "down"])
def test_fp16_grouped_gemm_reads_every_weight_from_its_place(pkg, hot):
    """One-hot tokens through the GEMM's gate/up and down boxes, 128 to each of two experts and all 256 through the shared MLP:
    output (token k, column h) is one weight of the matrix under test.  silu(64) = 64 and the other two matrices are constants or
    (scaled) identities, so up and down come out exactly; gate as silu(w), a rounding to fp16 (2^-11) and the fast exponential away."""
    D = 256
    rng = np.random.default_rng(44)
    eye, const = np.eye(D, dtype=np.float32), np.ones((D, D), dtype=np.float32)
    # gate, up, down around the matrix w under test: out[k][h] = silu(w[h][k]), w[h][k], w[h][k]
    others = {"gate": (None, const, eye), "up": (64 * const, None, eye), "down": (64 * const, eye / 64, None)}[hot]
    tests = [rng.integers(-512, 512, (D, D)).astype(np.float32) / (8192 if hot == "up" else 128) for _ in range(3)]      # all fp16 values
    full = [[w if m is None else m for m in others] for w in tests]
    slab = np.concatenate([m.reshape(-1) for e in full[:2] for m in e]).astype(np.float16).view(np.uint8)
    zero = np.zeros((D, D), dtype=np.float32)
    token = np.arange(D)
    inj = np.where(token[:, None] % 2 == np.arange(2)[None], 0.0, -1e4).astype(np.float32)
    x = torch.eye(D, dtype=torch.float16, device="cuda")
    for shared in (False, True):
        parts = full[2] if shared else [zero] * 3
        L = quant.LayerWeights(H=D, E=2, K=1, F=D, S=D, scaling=0.0 if shared else 1.0, router=np.zeros((2, D), np.uint16),
                               expert_qtype=quant.QTYPE_F16, expert_qweight=slab, expert_qscale=None,
                               **{n: quant.make_matrix(quant.QTYPE_F16, w) for n, w in zip(("shared_gate", "shared_up", "shared_down"), parts)})
        g = Layer(pkg, L, D)
        try:
            out = torch.zeros((D, D), dtype=torch.float16, device="cuda")
            g.ctx.layer_forward(0, x, D, out, injected_logits=dev(inj))
            g.ctx.synchronize()
        finally:
            g.close()
        w = np.stack([tests[2 if shared else k % 2][:, k] for k in token]).astype(np.float64)
        got = out.cpu().numpy().astype(np.float64)
        if hot == "gate":
            want = w / (1 + np.exp(-w))
            assert np.all(np.abs(got - want) <= 2.0 ** -10 * np.abs(want) + 2.0 ** -24), float(np.abs(got - want).max())
        else:
            assert np.array_equal(got, (64 * w if hot == "up" else w))


@pytest.mark.parametrize("pad", [16, 48, 128 * 128 * 2])
def test_fp16_slab_with_gaps_gives_the_packed_slabs_bits(pkg, pad):
    """Gaps of any multiple of 16 bytes between the projections: strides that are no multiples of one another, and ones that are
    multiples of a row but not of a matrix."""
    L, hidden, _ = make(43, dict(H=128, E=4, K=2, F=256, S=128), "f16", 40)
    outs, held = [], []
    for layer in (L, padded_slab_layer(L, pad_bytes=pad)):
        g = Layer(pkg, layer, 40)
        try:
            held.append(g.ctx.model_view_bytes)
            for n in (1, 3, 40):
                out = torch.zeros((n, L.H), dtype=torch.float16, device="cuda")
                g.ctx.layer_forward(0, dev(hidden[:n]), n, out)
                g.ctx.synchronize()
                outs.append(out)
        finally:
            g.close()
    assert held[0] == held[1]
    assert all(torch.equal(a, b) for a, b in zip(outs[:3], outs[3:]))


@pytest.mark.parametrize("n,K,E", [(31, 1, 8), (341, 3, 9), (512, 2, 8), (205, 5, 10), (1025, 1, 256), (1365, 6, 64), (1366, 6, 64),
                                   (1366, 6, 63), (1366, 6, 130)])
def test_dispatch_plan_at_step_edges(pkg, n, K, E):
    """Pair counts around a warp's step and a CTA's round, and around the 8192 pairs above which a context's plan takes the
    many-CTA form (for an even E up to 128); some experts without pairs, some ids out of range.  Both entry points: the
    allocation-free one always runs the one-CTA form."""
    rng = np.random.default_rng(n)
    ids = rng.integers(0, max(1, E - 2), size=(n, K)).astype(np.uint32)
    ids[rng.integers(0, n, 3), 0] = E + 1
    flat = ids.reshape(-1)
    order = np.argsort(flat, kind="stable")
    order = order[flat[order] < E]
    want_inv = np.full(n * K, 0xFFFFFFFF, dtype=np.uint32)
    want_inv[order] = np.arange(order.size, dtype=np.uint32)
    counts = np.bincount(flat[flat < E], minlength=E)
    L, _, _ = make(1, dict(H=64, E=E, K=K, F=64, S=64), "q8_0", 1)
    g = Layer(pkg, L, n)
    try:
        for plan in (pkg.ffi.dispatch_plan_noalloc, g.ctx.dispatch_plan):
            off = torch.zeros(E + 1, dtype=torch.int32).cuda()
            rows = torch.full((n * K,), -1, dtype=torch.int32).cuda()
            inv = torch.zeros(n * K, dtype=torch.int32).cuda()
            before = g.ctx.kernel_launches
            plan(dev(ids.view(np.int32)), n, K, E, off, rows, inv)
            torch.cuda.synchronize()
            if plan == g.ctx.dispatch_plan:
                assert g.ctx.kernel_launches - before == (3 if n * K > 8192 and E % 2 == 0 and E <= 128 else 1)
            assert np.array_equal(off.cpu().numpy(), np.concatenate([[0], np.cumsum(counts)]))
            assert np.array_equal(rows.cpu().numpy()[: order.size], order)
            assert np.array_equal(inv.cpu().numpy().view(np.uint32), want_inv)
    finally:
        g.close()


@pytest.mark.parametrize("n,E", [(1365, 64), (1366, 64), (1366, 63), (1366, 130)])
def test_grouped_gemm_with_tile_lists_of_either_plan(pkg, port, n, E):
    """Tile lists written by the one-CTA plan (up to 8192 pairs, or an odd E, or E above 128) and by the many-CTA one."""
    L, hidden, resid = make(800 + E, dict(H=128, E=E, K=6, F=128, S=128), "q8_0", n, bias="zipf")
    check_layer(pkg, port, L, hidden, resid, gemm=True)


@pytest.mark.parametrize("qname", ["q4_0", "q8_0"])
@pytest.mark.parametrize("n", [3, 4, 5, 16, 17])
def test_batched_decode_at_n_block_edges(pkg, port, qname, n):
    """Every token takes the same experts, so each item has n (or, above 16, 16 and n - 16) tokens: one to four blocks of four."""
    L, hidden, resid = make(500 + n, FULL, qname, n)
    hidden[:] = hidden[0]
    check_layer(pkg, port, L, hidden, resid)


@pytest.mark.parametrize("qname", ["q4_0", "q8_0"])
def test_batched_decode_gives_a_token_the_same_bits_in_every_batch(pkg, qname):
    """64 tokens in one call and in calls of 2, 3, 4, 5, 16 and 17: their experts' items hold one to sixteen tokens, one slice or
    two, and a sum in another order would show in some of the 81920 outputs."""
    L, hidden, _ = make(550, FULL, qname, 64)
    g = Layer(pkg, L, 64)
    try:
        x = dev(hidden).view(torch.float16)
        whole, parts = (torch.zeros((64, FULL["H"]), dtype=torch.float16, device="cuda") for _ in range(2))
        g.ctx.layer_forward(0, x, 64, whole)
        for size in (2, 3, 4, 5, 16, 17):
            parts.zero_()
            last = 64 // size * size
            for i in range(0, last, size):
                g.ctx.layer_forward(0, x[i:i + size], size, parts[i:i + size])
            g.ctx.synchronize()
            assert torch.equal(whole[:last].view(torch.int16), parts[:last].view(torch.int16)), size
    finally:
        g.close()


@pytest.mark.parametrize("qname,n", [("q4_0", 2), ("q8_0", 5), ("q4_0", 64)])
def test_batched_decode_with_the_norm_folded_in(pkg, qname, n):
    """The routing kernel's own RMSNorm equals the norm kernel followed by the plain call bit for bit."""
    L, hidden, _ = make(600 + n, FULL, qname, n)
    w = torch.rand(FULL["H"], device="cuda").add_(0.5).half()
    x = dev(hidden).view(torch.float16)
    g = Layer(pkg, L, n)
    try:
        folded, normed, plain = (torch.zeros((n, FULL["H"]), dtype=torch.float16, device="cuda") for _ in range(3))
        g.ctx.layer_forward_normed(0, x, w, 1e-6, n, folded)
        g.ctx.rmsnorm(x, w, 1e-6, n, FULL["H"], normed)
        g.ctx.layer_forward(0, normed, n, plain, residual=x)
        g.ctx.synchronize()
        assert torch.equal(folded, plain)
        with pytest.raises(pkg.UocrCudaError, match="RMSNorm"):
            g.ctx.layer_forward_normed(0, x, w, -1.0, n, folded)
    finally:
        g.close()


@pytest.mark.parametrize("qname,n", [("q4_0", 2), ("q8_0", 17), ("q4_0", 64)])
def test_batched_decode_with_the_norm_on_a_stream_at_an_8_byte_address(pkg, qname, n):
    """A stream that starts 8 bytes past a multiple of 16 takes the norm kernel (one launch more) and gives the same bits."""
    L, hidden, _ = make(620 + n, FULL, qname, n)
    w = torch.rand(FULL["H"], device="cuda").add_(0.5).half()
    x = dev(hidden).view(torch.float16)
    buf = torch.zeros(n * FULL["H"] + 8, dtype=torch.float16, device="cuda")
    off = (8 - buf.data_ptr()) % 16 // 2
    moved = buf[off:off + n * FULL["H"]].view(n, FULL["H"])
    moved.copy_(x)
    assert x.data_ptr() % 16 == 0 and moved.data_ptr() % 16 == 8
    g = Layer(pkg, L, n)
    try:
        outs, launches = [], []
        for rows in (x, moved):
            out, before = torch.zeros((n, FULL["H"]), dtype=torch.float16, device="cuda"), g.ctx.kernel_launches
            g.ctx.layer_forward_normed(0, rows, w, 1e-6, n, out)
            g.ctx.synchronize()
            outs.append(out)
            launches.append(g.ctx.kernel_launches - before)
        assert launches[1] == launches[0] + 1
        assert torch.equal(outs[0], outs[1])
    finally:
        g.close()


@pytest.mark.parametrize("qname,dims,n", [("f16", FULL, 2), ("f16", FULL, 3), ("f16", dict(H=2048, E=6, K=3, F=64, S=192), 9),
                                          ("q4_0", dict(H=192, E=5, K=2, F=64, S=320), 5), ("q8_0", dict(H=2048, E=5, K=2, F=192, S=64), 7)])
def test_matrix_vector_kernels_at_row_and_token_edges(pkg, port, qname, dims, n):
    """One, two, up to four and more tokens per expert, rows shorter than a warp's step and as long as the staging buffer, and
    activation rows that start at an address that is a multiple of two only."""
    L, hidden, resid = make(700 + n, dims, qname, n)
    check_layer(pkg, port, L, hidden, resid)
    g = Layer(pkg, L, n)
    try:
        odd = torch.zeros(n * dims["H"] + 1, dtype=torch.float16, device="cuda")[1:]
        odd.copy_(dev(hidden).view(torch.float16).reshape(-1))
        outs = [torch.zeros((n, dims["H"]), dtype=torch.float16, device="cuda") for _ in range(2)]
        g.ctx.layer_forward(0, dev(hidden).view(torch.float16), n, outs[0])
        g.ctx.layer_forward(0, odd, n, outs[1])
        g.ctx.synchronize()
        assert torch.equal(outs[0], outs[1])
    finally:
        g.close()
