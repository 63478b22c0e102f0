"""The nonzero-split multiply and the dense bit tiles at the sizes where they can go wrong: chunk and tile edges, rows
that cross many chunks, empty rows, ragged widths, unaligned operands, several thread blocks sharing a row panel."""
import pytest
import torch

from cagnet_b200 import _native, graphs, ops, partition as PP

pytestmark = pytest.mark.gpu
REL = 1e-5


def _close(got, want64):
    want64 = want64.double()
    err = float((got.double().cpu() - want64).abs().max())
    assert err <= REL * max(float(want64.abs().max()), 1e-30), err


def _dense64(b):
    return torch.sparse_coo_tensor(torch.stack([b.rows, b.cols]), b.vals.double(), (b.n_rows, b.n_cols))


@pytest.mark.parametrize("f", [1, 5, 16, 23, 41, 64, 65, 96, 100, 129, 300])
@pytest.mark.parametrize("lens", [[200], [1] * 70, [0, 31, 1, 0, 64, 33, 0], [65, 5000, 0, 1, 32, 32, 4000, 7], [3, 97] * 40 + [0]])
def test_split_multiply(f, lens):
    g = torch.Generator().manual_seed(f)
    n, m = len(lens), 6000
    rows = torch.repeat_interleave(torch.arange(n), torch.tensor(lens))
    cols = torch.cat([torch.sort(torch.randperm(m, generator=g)[:k])[0] for k in lens])
    blk = PP.Block(rows, cols, torch.randn(rows.numel(), generator=g), n, m)
    A = ops.CsrBlock.from_coo(blk.rows, blk.cols, blk.vals, n, m)
    A.max_row = -1                                   # as if unknown: the split form whatever the rows look like
    assert A.split is not None
    B, C0 = torch.randn(m, f, generator=g), torch.randn(n, f, generator=g)
    prod = torch.sparse.mm(_dense64(blk), B.double())
    for padded in (True, False):
        for beta in (0.0, 1.0):
            Bd = ops.to_padded(B.cuda()) if padded else B.cuda()
            Cd = ops.to_padded(C0.cuda()) if padded else C0.cuda().clone()
            ops.spmm(A, Bd, Cd, beta)
            _close(Cd, prod + beta * C0.double())
    wide = torch.full((n, f + 3), 7.0, device="cuda")             # a slice of a wider matrix, rows not 16-byte aligned
    ops.spmm(A, ops.to_padded(B.cuda()), wide[:, 1:f + 1], 0.0)
    _close(wide[:, 1:f + 1], prod)
    assert bool((wide[:, 0] == 7.0).all()) and bool((wide[:, f + 1:] == 7.0).all())


@pytest.mark.parametrize("nnz", [149999, 500000, 2000001])              # sizes at which the lane mapping changes
def test_split_multiply_lane_mappings(nnz):
    n, m = 3001, 5003
    g = torch.Generator(device="cuda").manual_seed(nnz)
    keys = torch.randperm(n * m, generator=g, device="cuda")[:nnz].sort()[0]
    rows, cols = keys // m, keys % m
    rows[:20000] = 0                                                       # one row of many chunks
    vals = torch.rand(nnz, generator=g, device="cuda")
    A = ops.CsrBlock.from_coo(rows, cols, vals, n, m)
    M = torch.sparse_coo_tensor(torch.stack([rows, cols]), vals.double(), (n, m))
    for f in (36, 64, 68, 96, 128, 132, 256, 600):
        B, C0 = torch.randn(m, f, generator=g, device="cuda"), torch.randn(n, f, generator=g, device="cuda")
        want = torch.sparse.mm(M, B.double())
        Bd, C = ops.to_padded(B), ops.to_padded(C0)
        ops.spmm(A, Bd, C, 1.0)
        _close(C, (want + C0.double()).cpu())
        ops.spmm(A, Bd, C, 0.0)
        _close(C, want.cpu())
        out = C0.clone()
        ops.spmm_gpu(rows.int(), cols.int(), vals, n, m, B, out)
        _close(out, (want + C0.double()).cpu())


@pytest.mark.parametrize("n,nnz,parts", [(700, 60000, 1), (4099, 600000, 1), (9001, 1500000, 3)])
def test_bit_tiles(n, nnz, parts):
    if not ops.integer_core_available():
        pytest.skip("library built without the tensor-core kernels")
    adj = graphs.add_self_loops(graphs.rmat_graph(n, target_nnz=nnz, seed=n), n)
    adj = torch.cat([adj, adj[:, :500]], dim=1)                    # some edges twice: those entries stay sparse
    blk = PP.fuse_columns(PP.oned_partition(0, parts, torch.zeros(n, 1), adj, True)[1])
    old = ops.configure_core(min_share=0.0, tile_nnz=1000, density_int=0.02)
    try:
        A = ops.CsrBlock.from_coo(blk.rows, blk.cols, blk.vals, blk.n_rows, n, row_scale=blk.row_scale, col_scale=blk.col_scale)
    finally:
        ops.configure_core(**old)
    assert A.tiles is not None
    bits = A.tiles.tile_bits.cpu().numpy().view("uint8")
    assert int(sum(bin(b).count("1") for b in bits.tolist())) + A.sparse.nnz == A.nnz
    M = _dense64(blk)
    for f in (1, 16, 17, 41, 64, 65, 128, 200, 602):
        g = torch.Generator().manual_seed(f)
        B, C0 = torch.randn(n, f, generator=g), torch.randn(blk.n_rows, f, generator=g)
        want = torch.sparse.mm(M, B.double()) + C0.double()
        Bd = ops.to_padded(B.cuda())
        if Bd.stride(0) > f:
            ops.base_buffer(Bd).view(-1, Bd.stride(0))[:, f:] = float("nan")
        C1, C2, C3 = ops.to_padded(C0.cuda()), ops.to_padded(C0.cuda()), C0.cuda().clone()
        ops.spmm(A, Bd, C1, 1.0)
        ops.spmm(A, Bd, C2, 1.0)
        ops.spmm(A, B.cuda(), C3, 1.0)                             # unaligned rows where f is not a multiple of 4
        _close(C1, want)
        _close(C3, want)
        assert torch.equal(C1, C2)
    assert _native.lib().cagnet_tile_core_error() == 0


@pytest.mark.parametrize("n,N,lo,hi", [(1, 1, 0, 1), (33, 7, 0, 7), (300, 41, 0, 41), (257, 256, 0, 256), (500, 20, 20, 40)])
def test_fused_loss_and_adam(n, N, lo, hi):
    """Loss, gradient before the log-softmax and one Adam step against fp64 autograd and torch.optim.Adam."""
    import ctypes
    L, g = _native.lib(), torch.Generator().manual_seed(n)
    z = torch.randn(n, N, generator=g)
    y = torch.randint(0, 2 * N, (n,), generator=g)
    mask = torch.rand(n, generator=g) < 0.7
    mask[0] = True
    y[0] = lo
    hit = mask & (y >= lo) & (y < hi)
    z64 = z.double().requires_grad_(True)
    want = -torch.log_softmax(z64, dim=1)[hit, (y - lo)[hit]].sum() / n
    want.backward()
    logp, dz = ops.log_softmax(ops.to_padded(z.cuda())), ops.empty_padded(n, N, "cuda")
    ws = torch.empty(L.cagnet_nll_workspace_bytes(n), dtype=torch.uint8, device="cuda")
    parts = ctypes.c_int32()
    yd, md = y.cuda(), mask.cuda().view(torch.uint8)
    _native.check(L.cagnet_nll_softmax_bwd_f32(logp.data_ptr(), logp.stride(0), yd.data_ptr(), md.data_ptr(), n, N, lo, hi, float(n),
                                               dz.data_ptr(), dz.stride(0), ctypes.byref(parts), ws.data_ptr(), ws.numel(), None))
    _close(dz, z64.grad)
    w = [torch.randn(*k, generator=g).cuda() for k in ((n, 3), (5, N))]
    ref = [torch.nn.Parameter(t.clone()) for t in w]
    opt = torch.optim.Adam(ref, lr=0.01)
    state = [[torch.zeros_like(t), torch.zeros_like(t)] for t in w]
    loss = torch.empty((), device="cuda")
    for step in (1, 2, 3):
        partials = [torch.randn(11, 3, n, generator=g).cuda(), torch.randn(3, 5, N, generator=g).cuda()]      # the first transposed
        sums = [_native.TnSum(d.data_ptr(), d.size(0), d.size(1), d.size(2), k) for d, k in zip(partials, (1, 0))]
        grads = [torch.full_like(t, float("nan")) for t in w]
        ptr = [x for t, s, d, q in zip(w, state, grads, sums) for x in (ctypes.addressof(q), d.data_ptr(), t.data_ptr(), s[0].data_ptr(), s[1].data_ptr())]
        _native.check(L.cagnet_epoch_tail_f32(*ptr, 0.01, 0.9, 0.999, 1e-8, step, ws.data_ptr(), parts.value, float(n), loss.data_ptr(), None))
        _close(grads[0], partials[0].double().sum(0).t().cpu())
        _close(grads[1], partials[1].double().sum(0).cpu())
        for p, d in zip(ref, grads):
            p.grad = d.clone()
        opt.step()
    for t, p in zip(w, ref):
        _close(t, p.detach().cpu())
    assert abs(float(loss) - float(want)) <= 1e-5 * max(abs(float(want)), 1e-6)


@pytest.mark.parametrize("n,K,N", [(9472, 304, 16), (9601, 350, 41), (20001, 130, 100), (40003, 16, 256), (40003, 64, 80), (70000, 602, 10),
                                   (33000, 33, 65), (19000, 64, 200), (30011, 96, 8)])
def test_tensor_core_products(n, K, N):
    """X.W and H^T.G at sizes that the tcgen05 kernels take, tile remainders in every direction, against fp64: as close as
    fp32 multiply-adds come (one bf16 term would be 2e-3 off, two 1e-5), bit-reproducible, pad columns never read or written."""
    g = torch.Generator(device="cuda").manual_seed(n)
    X, W = torch.randn(n, K, generator=g, device="cuda"), torch.randn(K, N, generator=g, device="cuda")
    aux, Z0 = torch.randn(n, N, generator=g, device="cuda"), torch.randn(n, N, generator=g, device="cuda")
    Xd = ops.to_padded(X)
    if Xd.stride(0) > K:
        ops.base_buffer(Xd).view(-1, Xd.stride(0))[:, K:] = float("nan")
    want = X.double() @ W.double()

    def close(got, ref):
        assert float((got.double() - ref).norm()) <= 1e-6 * float(ref.norm())
    for trans, w in ((False, W), (True, W.t().contiguous())):
        Z = ops.gemm_nn(Xd, w, trans)
        close(Z, want)
        assert torch.equal(Z, ops.gemm_nn(Xd, w, trans))
    close(ops.gemm_nn(Xd, W, False, ops.EPI_RELU), torch.relu(want))
    close(ops.gemm_nn(Xd, W, False, ops.EPI_RELU_MASK, aux=ops.to_padded(aux)), want * (aux > 0))
    close(ops.gemm_nn(Xd, W, False, ops.EPI_ACCUMULATE, out=ops.to_padded(Z0)), want + Z0.double())
    wide = torch.full((n, N + 5), 7.0, device="cuda")
    ops.gemm_nn(Xd, W, False, ops.EPI_NONE, out=wide[:, 1:N + 1])          # rows of Z not 16-byte aligned
    close(wide[:, 1:N + 1], want)
    assert bool((wide[:, 0] == 7.0).all()) and bool((wide[:, N + 1:] == 7.0).all())
    if N <= 64 or N <= 256 and K <= 64:
        out = ops.empty_padded(n, N, "cuda")
        epi = ops.EPI_LOG_SOFTMAX if N <= 64 else 5
        _native.check(_native.lib().cagnet_gemm_nn_f32(Xd.data_ptr(), Xd.stride(0), W.data_ptr(), N, 0, out.data_ptr(), out.stride(0), n, K,
                                                       N, epi, None, 0, None))
        close(out, torch.log_softmax(want, dim=1))
    Gd = ops.to_padded(Z0)
    if Gd.stride(0) > N:
        ops.base_buffer(Gd).view(-1, Gd.stride(0))[:, N:] = float("nan")
    grad = ops.gemm_tn(Xd, Gd)
    close(grad, X.double().t() @ Z0.double())
    assert torch.equal(grad, ops.gemm_tn(Xd, Gd))
    assert _native.lib().cagnet_tile_core_error() == 0


@pytest.mark.parametrize("n,K,N,lo", [(70, 12, 7, 0), (3001, 100, 30, 2), (5003, 20, 130, 0), (60001, 16, 41, 0), (60001, 40, 64, 3),
                                       (40003, 100, 30, 0), (40003, 16, 97, 0), (40003, 64, 256, 5)])
def test_product_with_loss(n, K, N, lo):
    """log_softmax(X.W), its masked NLL and the gradient before the log-softmax from one call, against fp64."""
    import ctypes
    L, g, hi = _native.lib(), torch.Generator(device="cuda").manual_seed(n + N), lo + N - 1
    X, W = torch.randn(n, K, generator=g, device="cuda"), torch.randn(K, N, generator=g, device="cuda")
    y = torch.randint(0, hi + 3, (n,), generator=g, device="cuda")
    mask = torch.rand(n, generator=g, device="cuda") < 0.6
    want = torch.log_softmax(X.double() @ W.double(), dim=1)
    hit = mask & (y >= lo) & (y < hi)
    grad = want.exp()
    grad[hit, (y - lo)[hit]] -= 1
    grad = torch.where(hit[:, None], grad / n, torch.zeros_like(grad))
    ws, parts, launches = torch.zeros(L.cagnet_nll_workspace_bytes(n) // 4, device="cuda"), ctypes.c_int32(), ctypes.c_int32()
    for make in (ops.empty_padded, lambda n, N, d: torch.full((n, N + 1), 7.0, device=d)[:, 1:]):         # rows on 16 bytes, and not
        logp, dz = make(n, N, "cuda"), make(n, N, "cuda")
        Xd = ops.to_padded(X)
        _native.check(L.cagnet_gemm_nll_f32(Xd.data_ptr(), Xd.stride(0), W.data_ptr(), N, n, K, N, y.data_ptr(), mask.data_ptr(), lo, hi,
                                            float(n), logp.data_ptr(), logp.stride(0), dz.data_ptr(), dz.stride(0), ctypes.byref(parts),
                                            ctypes.byref(launches), ws.data_ptr(), ws.numel() * 4, None))
        assert float((logp.double() - want).norm()) <= 1e-6 * float(want.norm())
        assert float((dz.double() - grad).norm()) <= 1e-6 * float(grad.norm())
        total = want[hit, (y - lo)[hit]].sum()
        assert abs(float(ws[:parts.value].double().sum() - total)) <= 1e-6 * abs(float(total))
        z = make(n, N, "cuda").copy_(X @ W)                                   # the same from the logits, in place
        dz.fill_(9.0)
        _native.check(L.cagnet_log_softmax_nll_f32(z.data_ptr(), z.stride(0), n, N, y.data_ptr(), mask.data_ptr(), lo, hi, float(n),
                                                   z.data_ptr(), z.stride(0), dz.data_ptr(), dz.stride(0), ctypes.byref(parts),
                                                   ws.data_ptr(), ws.numel() * 4, None))
        assert float((z.double() - want).norm()) <= 1e-6 * float(want.norm())
        assert float((dz.double() - grad).norm()) <= 1e-6 * float(grad.norm())
        assert abs(float(ws[:parts.value].double().sum() - total)) <= 1e-6 * abs(float(total))
    assert launches.value == (2 if N <= 64 <= K and n < 40000 else 1) and L.cagnet_tile_core_error() == 0
