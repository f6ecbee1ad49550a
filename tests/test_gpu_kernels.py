"""sm_100a kernels against plain PyTorch fp32 references of the same op."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return ((a.float() - b.float()).norm() / (b.float().norm() + 1e-12)).item()


@pytest.fixture(scope="module")
def cb():
    from dawn_srw_b200.ops import cuda_backend as CB
    CB.ext()          # must load: a missing extension is an error on a GPU box
    return CB


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("shape", [(128, 128, 64), (384, 520, 320), (200, 1000, 136), (1000, 392, 200)])
@pytest.mark.parametrize("bn", [128, 256])
def test_gemm_against_fp32_matmul(cb, a_mn, b_mn, shape, bn):
    M, N, K = shape
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(M + N + K)
    A = torch.randn(M, K, device=dev, generator=g).bfloat16()
    B = torch.randn(N, K, device=dev, generator=g).bfloat16()
    ref = A.float() @ B.float().t()
    As = A.t().contiguous() if a_mn else A
    Bs = B.t().contiguous() if b_mn else B
    out = cb.gemm(As, a_mn, Bs, b_mn, out_dtype=torch.float32, block_n=bn)
    torch.cuda.synchronize()
    assert _rel(out, ref) < 1e-5
    cb.check_status()


def test_gemm_epilogue_options(cb):
    dev = torch.device("cuda")
    A = torch.randn(300, 264, device=dev).bfloat16()
    B = torch.randn(520, 264, device=dev).bfloat16()
    rs = torch.rand(300, device=dev) + 0.5
    bias = torch.randn(520, device=dev)
    ref = (A.float() @ B.float().t()) * rs[:, None] * 0.5 + bias
    out = cb.gemm(A, False, B, False, out_dtype=torch.bfloat16, alpha=0.5, row_scale=rs, bias=bias)
    assert _rel(out, ref) < 5e-3
    acc = torch.ones(300, 520, device=dev)
    cb.gemm(A, False, B, False, out=acc, accumulate=True)          # TMA reduce-add
    assert _rel(acc, A.float() @ B.float().t() + 1.0) < 1e-5
    # a second accumulation into the same buffer adds again
    cb.gemm(A, False, B, False, out=acc, accumulate=True)
    assert _rel(acc, 2 * (A.float() @ B.float().t()) + 1.0) < 1e-5
    # few output tiles with a long K: the launcher cuts K and the splits meet in the reduce-add
    A2 = torch.randn(8192, 304, device=dev).bfloat16()      # stored [K, M]
    B2 = torch.randn(8192, 264, device=dev).bfloat16()      # stored [K, N]
    acc2 = torch.full((304, 264), 0.5, device=dev)
    cb.gemm(A2, True, B2, True, out=acc2, accumulate=True)
    assert _rel(acc2, A2.float().t() @ B2.float() + 0.5) < 1e-5
    cb.check_status()


@pytest.mark.parametrize("M,N,K,a_mn", [(8, 384, 25200, False), (6, 1280, 10400, False),
                                        (231, 384, 25200, False), (256, 256, 10400, True),
                                        (128, 128, 25200, True)])
def test_accumulating_gemm_whose_k_tiles_do_not_divide_into_splits(cb, M, N, K, a_mn):
    """K tiles that leave the last of the wanted splits empty (163 = 18 * 9 + 1, not 20 * 9): a
    split without K tiles would add the previous launch's accumulators.  fp32 accumulation of
    exact bf16 products in any order is within K * 2^-24 of the row norms' product, i.e. far
    below 1e-5 of a random result's norm; a stale accumulator is of the order of one."""
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(K + M)
    A = torch.randn(M, K, device=dev, generator=g).bfloat16()
    B = torch.randn(K, N, device=dev, generator=g).bfloat16()
    ref = A.double() @ B.double()
    As = A.t().contiguous() if a_mn else A
    big = torch.randn(512, 1024, device=dev, generator=g).bfloat16()
    for _ in range(2):
        cb.gemm(big, False, big, False)                      # leaves values in the accumulators
        out = torch.zeros(M, N, device=dev)
        cb.gemm(As, a_mn, B, True, out=out, accumulate=True)
        assert _rel(out, ref) < 1e-5
    cb.check_status()


@pytest.mark.parametrize("M", [1, 32, 128])
def test_engine_gemm_with_few_rows(cb, M):
    """Up to 128 rows: single-CTA tiles, and the long K of a decode-step write GEMM is cut
    into splits that meet in the reduce-add epilogue."""
    dev = torch.device("cuda")
    torch.manual_seed(M)
    for K, N in ((6400, 1280), (20000, 384), (72, 520)):
        A = torch.randn(M, K, device=dev).bfloat16()
        Bt = torch.randn(K, N, device=dev).bfloat16()         # stored [K, N]: MN-major operand
        ref = A.float() @ Bt.float()
        y = torch.full((M, N), 0.25, device=dev)
        cb.gemm(A, False, Bt, True, out=y, accumulate=True)
        assert _rel(y, ref + 0.25) < 1e-5
        out = cb.gemm(A, False, Bt.t().contiguous(), False, out_dtype=torch.bfloat16)
        assert _rel(out, ref) < 5e-3
    cb.check_status()


@pytest.mark.parametrize("kind", [0, 1, 2])
@pytest.mark.parametrize("T", [1, 7, 128])
def test_forward_gate_kernel_with_few_rows(cb, kind, T):
    """Decode shapes run the 256-wide gate kernel on single CTAs (128 x 256 tiles)."""
    from dawn_srw_b200.ops.gates import GateSpec, gate_forward
    dev = torch.device("cuda")
    torch.manual_seed(10 * T + kind)
    U, r, D = 3001, 128, 384
    spec = GateSpec(kind=kind)
    nz = torch.nn.functional.normalize
    h, x = torch.randn(T, r, device=dev).bfloat16(), torch.randn(T, D, device=dev).bfloat16()
    emb, read = (nz(torch.randn(U, d, device=dev), dim=-1).bfloat16() for d in (r, D))
    s = h.float() @ emb.float().t()
    mu, sd = s.mean(-1, keepdim=True), s.std(-1, unbiased=False, keepdim=True) + 1e-8
    tau = mu + 0.3 * sd
    g, dt, _ = gate_forward(spec, s, tau, sd)
    Up = (U + 7) // 8 * 8
    p = torch.zeros(T, Up, device=dev, dtype=torch.bfloat16)
    den = torch.zeros(T, device=dev)
    e, st, gl = cb.ext(), cb.status_word(dev), cb._gate_list(spec)
    e.srw_fwd_gate_xr(h, emb, x, read, p, None, tau.squeeze(-1).contiguous(),
                      (1 / sd).squeeze(-1).contiguous(), None, den, None, None, None, gl, st,
                      *cb.NO_GATHER)
    assert _rel(p[:, :U], g * (x.float() @ read.float().t())) < 6e-3
    assert _rel(den, dt.sum(-1)) < 1e-4
    cb.check_status()


@pytest.mark.parametrize("kind", [0, 1, 2])
@pytest.mark.parametrize("N,D,r", [(1, 1280, 256), (2, 1280, 256), (3, 384, 128), (4, 1024, 256),
                                   (2, 2048, 384)])
def test_streaming_pool_op_for_a_few_rows(cb, kind, N, D, r):
    """The SIMT decode kernel (one pass over the pool, normalisation and scale applied by its
    second kernel) against the fp32 formula with p rounded to bf16."""
    from dawn_srw_b200.ops.gates import GateSpec, gate_forward
    dev = torch.device("cuda")
    torch.manual_seed(100 * N + kind)
    U = 5003
    spec = GateSpec(kind=kind)
    nz = torch.nn.functional.normalize
    h, x = torch.randn(N, r, device=dev).bfloat16(), torch.randn(N, D, device=dev).bfloat16()
    Up = (U + 7) // 8 * 8
    emb, read, write = (torch.zeros(Up, d, device=dev, dtype=torch.bfloat16) for d in (r, D, D))
    for t, d in ((emb, r), (read, D), (write, D)):
        t[:U] = nz(torch.randn(U, d, device=dev), dim=-1).bfloat16()
    s = h.float() @ emb[:U].float().t()
    mu, sd = s.mean(-1, keepdim=True), s.std(-1, unbiased=False, keepdim=True) + 1e-8
    tau = mu + 0.8 * sd                                   # most units of the relu-type gates are off
    g, dt, _ = gate_forward(spec, s, tau, sd)
    p = (g * (x.float() @ read[:U].float().t())).bfloat16().float()
    scale = torch.tensor(1.7, device=dev)
    ref = (p @ write[:U].float()) * (scale / dt.sum(-1).clamp(min=1.0))[:, None]
    e = cb.ext()
    out, den = e.srw_rows(h, x, tau.squeeze(-1).contiguous(), (1 / sd).squeeze(-1).contiguous(),
                          emb[:U], read[:U], write[:U], None, cb._gate_list(spec), 1.0, scale.reshape(1))
    assert _rel(den, dt.sum(-1)) < 1e-4
    assert _rel(out, ref) < 3e-3
    out2, _ = e.srw_rows(h, x, tau.squeeze(-1).contiguous(), (1 / sd).squeeze(-1).contiguous(),
                         emb[:U], read[:U], write[:U], None, cb._gate_list(spec), 1.7, None)
    assert _rel(out, out2) < 1e-5       # the blocks' partial sums meet in a different order


@pytest.mark.parametrize("M", [1, 2, 3, 4])
def test_few_row_gemv_path_of_the_gemm_wrapper(cb, M):
    dev = torch.device("cuda")
    torch.manual_seed(M)
    for K, N in ((1280, 776), (384, 30522), (2048, 1283)):
        x = torch.randn(M, K, device=dev).bfloat16()
        Np = (N + 7) // 8 * 8
        w = torch.randn(Np, K, device=dev).bfloat16()[:N]
        bias = torch.randn(N, device=dev)
        ref = x.float() @ w.float().t() + bias
        out = cb.gemm(x, False, w, False, out_dtype=torch.float32, bias=bias)
        assert out.shape == (M, N) and _rel(out, ref) < 1e-5
    cb.check_status()


def test_decode_attention_kernel_extends_the_cache_and_matches_torch(cb):
    from dawn_srw_b200.ops import reference as R
    dev = torch.device("cuda")
    torch.manual_seed(11)
    B, H, dh, S = 3, 4, 80, 96
    ck, cv = torch.randn(B, H, S, dh, device=dev), torch.randn(B, H, S, dh, device=dev)
    be = cb.CudaBackend()
    for pos in (0, 5, S - 1):
        q, k, v = (torch.randn(B, H * dh, device=dev) for _ in range(3))
        ck2, cv2 = ck.clone(), cv.clone()
        ck2[:, :, pos] = k.view(B, H, dh)
        cv2[:, :, pos] = v.view(B, H, dh)
        ref = R.cached_attention(q.view(B, H, 1, dh), ck2, cv2, pos + 1).reshape(B, H * dh)
        c1, c2 = ck.clone(), cv.clone()
        out = be.decode_attention(q, k, v, c1, c2, torch.tensor([pos], device=dev), H)
        assert torch.equal(c1, ck2) and torch.equal(c2, cv2)
        assert _rel(out, ref) < 1e-5


@pytest.mark.parametrize("B,H,dh,S", [(1, 16, 80, 512), (1, 2, 128, 1000), (6, 16, 128, 512), (5, 3, 36, 100),
                                      (40, 16, 64, 70), (2, 2, 20, 40), (3, 1, 30, 64)])
def test_decode_attention_over_split_positions(cb, B, H, dh, S):
    """Clusters of one to eight CTAs, groups without a position of their own, head rows that
    are no multiple of the lanes' chunks, and (dh = 30) the kernel for unaligned rows.  fp32
    throughout: the two sides differ by the order of the sums."""
    from dawn_srw_b200.ops import reference as R
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(S)
    rn = lambda *s: torch.randn(*s, device=dev, generator=g)
    ck, cv = rn(B, H, S, dh), rn(B, H, S, dh)
    be = cb.CudaBackend()
    for pos in (0, 1, 31, 33, S // 2, S - 1):
        q, k, v = rn(B, H * dh), rn(B, H * dh), rn(B, H * dh)
        ck[:, :, pos], cv[:, :, pos] = 7.0, float("nan")       # the call has to overwrite the slot
        out = be.decode_attention(q, k, v, ck, cv, torch.tensor([pos], device=dev), H)
        assert torch.equal(ck[:, :, pos].reshape(B, -1), k) and torch.equal(cv[:, :, pos].reshape(B, -1), v)
        ref = R.cached_attention(q.view(B, H, 1, dh), ck, cv, pos + 1).reshape(B, H * dh)
        assert _rel(out, ref) < 1e-5


def test_score_statistics_of_a_few_rows(cb):
    """The one-launch statistics kernel of the generation path against fp32 torch."""
    from dawn_srw_b200.ops.score_stats import score_stats_rows
    dev = torch.device("cuda")
    torch.manual_seed(3)
    T, R, r, U = 5, 2, 256, 3000
    emb = torch.nn.functional.normalize(torch.randn(U, r, device=dev), dim=-1)
    gram, esum = emb.t() @ emb, emb.sum(0)
    big = torch.randn(T, 3 * r + 8, device=dev)
    h = big[:, :2 * r].view(T, R, r)                          # strided view, as the router emits it
    off = torch.randn(T, 3, device=dev)[:, :2]
    tau, isd, hb = score_stats_rows(h, off, gram, esum, U)
    hq = h.bfloat16().float().transpose(0, 1).reshape(R * T, r)
    s = hq @ emb.t()
    mu, sd = s.mean(-1), s.std(-1, unbiased=False) + 1e-8
    assert torch.equal(hb.float(), hq)
    assert _rel(isd, 1 / sd) < 1e-4 and _rel(tau, mu + off.t().reshape(-1) * sd) < 1e-4


@pytest.mark.parametrize("kind", [0, 1, 2])
@pytest.mark.parametrize("dims", [(256, 384, 128, 384), (300, 1580, 128, 384), (130, 197, 64, 256),
                                  (300, 2504, 128, 384), (520, 4099, 64, 256), (260, 777, 64, 256)])   # U >= 512: 256-wide tiles
def test_gate_kernels(cb, kind, dims):
    from dawn_srw_b200.ops.gates import GateSpec, gate_backward, gate_forward
    T, U, r, D = dims
    dev = torch.device("cuda")
    spec = GateSpec(kind=kind)
    nz = torch.nn.functional.normalize
    torch.manual_seed(T + U + kind)
    h = torch.randn(T, r, device=dev).bfloat16()
    emb = nz(torch.randn(U, r, device=dev), dim=-1).bfloat16()
    x = torch.randn(T, D, device=dev).bfloat16()
    read = nz(torch.randn(U, D, device=dev), dim=-1).bfloat16()
    write = nz(torch.randn(U, D, device=dev), dim=-1).bfloat16()
    s = h.float() @ emb.float().t()
    mu, sd = s.mean(-1, keepdim=True), s.std(-1, unbiased=False, keepdim=True) + 1e-8
    tau = mu + 0.3 * sd
    g, dt, _ = gate_forward(spec, s, tau, sd)
    xr = x.float() @ read.float().t()
    Up = (U + 7) // 8 * 8
    p = torch.zeros(T, Up, device=dev, dtype=torch.bfloat16)
    den, gs = torch.zeros(T, device=dev), torch.zeros(T, device=dev)
    alive = torch.zeros(U, device=dev, dtype=torch.uint8)
    e, st, gl = cb.ext(), cb.status_word(dev), cb._gate_list(spec)
    tau_c, isd_c = tau.squeeze(-1).contiguous(), (1 / sd).squeeze(-1).contiguous()
    e.srw_fwd_gate(h, emb, x, read, p, tau_c, isd_c, den, gs, alive, None, gl, st)
    assert _rel(p[:, :U], g * xr) < 6e-3
    assert _rel(den, dt.sum(-1)) < 1e-4 and _rel(gs, g.sum(-1)) < 1e-4
    assert torch.equal(alive.bool(), g.max(0).values >= spec.dead_threshold)
    dy = (torch.randn(T, D, device=dev) * 0.1).bfloat16()
    dden = torch.randn(T, device=dev) * 0.01
    dp = dy.float() @ write.float().t()
    ds_ref, dtau_ref, _ = gate_backward(spec, s, tau, sd, dp * xr, dden[:, None])
    pb, dxr, ds = (torch.zeros_like(p) for _ in range(3))
    dtau, dsz = torch.zeros(T, device=dev), torch.zeros(T, device=dev)
    e.srw_bwd_gate(h, emb, x, read, dy, write, pb, dxr, ds, tau_c, isd_c, dden, dtau, dsz, gl, st)
    assert _rel(pb[:, :U], g * xr) < 6e-3 and _rel(dxr[:, :U], dp * g) < 6e-3
    assert _rel(ds[:, :U], ds_ref) < 1e-2 and _rel(dtau, dtau_ref.squeeze(-1)) < 4e-3  # gate coefficients are held as bf16
    if kind == 1:
        # the sigma-path reduction is recovered from ds.emb and dtau instead of a kernel output
        dh = ds[:, :U].float() @ emb.float()
        dsz_id = isd_c * ((h.float() * dh).sum(-1) + tau_c * dtau)
        assert _rel(dsz_id, (ds_ref * (s - tau) / sd).sum(-1)) < 2e-2
    cb.check_status()


@pytest.mark.parametrize("kind", [0, 1, 2])
@pytest.mark.parametrize("dims", [(300, 2504, 128, 384), (520, 4099, 64, 256), (260, 777, 64, 256),
                                  (1000, 3000, 256, 1280), (700, 2600, 384, 2048)])   # 400M / 1B widths
def test_gate_kernels_with_kept_read_scalars(cb, kind, dims):
    """The forward kernel also writes xr = x . read^T; the backward gate step then
    is one launch on S and DP that reads xr back (and may overwrite it with p)."""
    from dawn_srw_b200.ops.gates import GateSpec, gate_backward, gate_forward
    T, U, r, D = dims
    dev = torch.device("cuda")
    spec = GateSpec(kind=kind)
    nz = torch.nn.functional.normalize
    gen = torch.Generator(device=dev).manual_seed(T + U)
    rn = lambda *s: torch.randn(*s, device=dev, generator=gen)
    h, x = rn(T, r).bfloat16(), rn(T, D).bfloat16()
    emb, read, write = (nz(rn(U, d), dim=-1).bfloat16() for d in (r, D, D))
    s = h.float() @ emb.float().t()
    mu, sd = s.mean(-1, keepdim=True), s.std(-1, unbiased=False, keepdim=True) + 1e-8
    tau = mu + 0.3 * sd
    g, dt, _ = gate_forward(spec, s, tau, sd)
    xr_ref = x.float() @ read.float().t()
    Up = (U + 7) // 8 * 8
    p = torch.zeros(T, Up, device=dev, dtype=torch.bfloat16)
    xr = torch.full((T, Up), float("nan"), device=dev, dtype=torch.bfloat16)
    den = torch.zeros(T, device=dev)
    e, st, gl = cb.ext(), cb.status_word(dev), cb._gate_list(spec)
    assert e.srw_wide_tiles(U)
    tau_c, isd_c = tau.squeeze(-1).contiguous(), (1 / sd).squeeze(-1).contiguous()
    e.srw_fwd_gate_xr(h, emb, x, read, p, xr, tau_c, isd_c, None, den, None, None, None, gl, st, *cb.NO_GATHER)
    assert _rel(p[:, :U], g * xr_ref) < 6e-3 and _rel(xr[:, :U], xr_ref) < 4e-3
    assert _rel(den, dt.sum(-1)) < 1e-4
    dy = (rn(T, D) * 0.1).bfloat16()
    dden = rn(T) * 0.01
    dp = dy.float() @ write.float().t()
    xr_q = xr[:, :U].float()                       # what the backward kernel actually reads
    ds_ref, dtau_ref, _ = gate_backward(spec, s, tau, sd, dp * xr_q, dden[:, None])
    dxr, ds = torch.zeros_like(p), torch.zeros_like(p)
    dtau = torch.zeros(T, device=dev)
    e.srw_bwd_gate_xr(h, emb, dy, write, xr, xr, dxr, ds, tau_c, isd_c, dden, None, dtau, gl, st,
                      *cb.NO_GATHER)                        # p overwrites xr in place
    assert _rel(xr[:, :U], g * xr_q) < 6e-3 and _rel(dxr[:, :U], dp * g) < 6e-3
    assert _rel(ds[:, :U], ds_ref) < 8e-3 and _rel(dtau, dtau_ref.squeeze(-1)) < 4e-3
    cb.check_status()


@pytest.mark.parametrize("version", ["spatial-r1-v3.9.4", "spatial-r1-v4.0.1", "spatial-r1-v4.1"])
@pytest.mark.parametrize("dims", [(300, 1, 1580, 128, 384), (256, 2, 777, 64, 256)])
def test_srw_op_forward_backward_against_fp32_oracle(cb, version, dims):
    """Inputs are rounded to bf16 first so both paths see the same values; what
    remains is the bf16 rounding of the gated operand tiles."""
    from dawn_srw_b200.ops.backend import ParallelCtx, ReferenceBackend
    from dawn_srw_b200.ops.gates import gate_spec_for
    T, R, U, r, D = dims
    dev = torch.device("cuda")
    torch.manual_seed(11)
    spec = gate_spec_for(version)
    rb, kb = ReferenceBackend(torch.float32), cb.CudaBackend()
    q = lambda t: t.bfloat16().float()
    nz = torch.nn.functional.normalize
    emb, read, write = (torch.randn(U, d, device=dev) for d in (r, D, D))
    if not spec.normalize_pool:
        emb, read, write = q(nz(emb, dim=-1)), q(nz(read, dim=-1)), q(nz(write, dim=-1))
    x, h = q(torch.randn(T, D, device=dev)), q(torch.randn(T, R, r, device=dev))
    off = torch.randn(T, R, device=dev) * 0.3 - 0.3
    w = torch.randn(T, R, D, device=dev)
    res = {}
    for name, be in (("ref", rb), ("cuda", kb)):
        ps = [t.clone().requires_grad_(True) for t in (emb, read, write, x, h, off)]
        sc = torch.tensor(1.7, device=dev, requires_grad=True)         # learnable pool scale
        pool = be.prepare_pool(ps[0], ps[1], ps[2], spec, ParallelCtx())
        out = be.srw(ps[3], ps[4], ps[5], pool, spec, pctx=ParallelCtx(), want_diag=False,
                     out_scale=sc)
        ((out.stacked() * w).sum() + 3.0 * out.lb + 2.0 * out.dead_penalty).backward()
        res[name] = [out.stacked().detach(), out.lb.detach()] + [p.grad for p in ps] + [sc.grad]
    names = ["out", "lb", "demb", "dread", "dwrite", "dx", "dh", "doff", "dscale"]
    tol = {"out": 6e-3, "lb": 2e-3, "dread": 8e-3, "dwrite": 8e-3, "dx": 8e-3, "dscale": 5e-2}   # dscale: a scalar sum with heavy cancellation
    # gradients that flow through d(gate)/d(score): the bf16 rounding of the
    # (normalised) emb moves a few scores across the gate's kink, so these are
    # compared loosely here; tests/test_gates_and_srw.py and test_gate_kernels
    # check the same math tightly
    sharp = 0.08
    for n, a, b in zip(names, res["cuda"], res["ref"]):
        if n == "dscale":
            # one scalar, sum_t <d_out, out> / scale, with heavy cancellation between tokens:
            # compare against the size of the summed terms instead of the sum
            terms = float((res["ref"][0].abs() * w.abs()).sum() / 1.7)
            assert abs(float(a) - float(b)) < 2e-3 * terms, (n, float(a), float(b), terms)
            continue
        assert _rel(a, b) < tol.get(n, sharp), (n, _rel(a, b))
    cb.check_status()


@pytest.mark.parametrize("dims", [(300, 1, 128, 2600), (129, 2, 256, 6400), (64, 1, 384, 1000)])
def test_score_statistics_kernels(cb, dims):
    """tau, 1/sigma, column sums and all gradients of the Gram-matrix statistics:
    engine GEMMs + row kernels against the same node in plain fp32 torch on the CPU."""
    from dawn_srw_b200.ops.score_stats import score_stats
    T, R, r, U = dims
    torch.manual_seed(T)
    emb = torch.nn.functional.normalize(torch.randn(U, r), dim=-1).bfloat16().float()
    h0 = torch.randn(T, R, r).bfloat16().float()
    h0[3, 0] = 0.0                                   # a zero row sits on the variance floor
    off0 = torch.randn(T, R) * 0.4
    wt, wi, wh = torch.randn(T, R), torch.randn(T, R) * 1e-2, torch.randn(r)
    wb = torch.randn(T, R, r).bfloat16()
    out = {}
    for dev in ("cpu", "cuda"):
        leaf = lambda t: t.detach().clone().to(dev).requires_grad_(True)
        h, off = leaf(h0), leaf(off0)
        gram, esum = leaf(emb.t() @ emb), leaf(emb.sum(0))
        tau, isd, hsum, hb = score_stats(h, off, gram, esum, U)
        ((tau * wt.to(dev)).sum() + (isd * wi.to(dev)).sum() + (hsum * wh.to(dev)).sum()
         + (hb.float() * wb.to(dev).float()).sum()).backward()
        out[dev] = [t.detach().cpu() for t in (tau, isd, hsum, hb.float(), h.grad, off.grad,
                                               gram.grad, esum.grad)]
    cb.check_status()
    names = ("tau", "isd", "hsum", "hb", "dh", "doff", "dgram", "desum")
    for n, a, b in zip(names, out["cuda"], out["cpu"]):
        assert torch.isfinite(a).all(), n
        tol = 2e-2 if n == "dgram" else 2e-3          # dG multiplies bf16-rounded d_var * h
        assert _rel(a, b) < tol, (n, _rel(a, b))


@pytest.mark.parametrize("version", ["spatial-r1-v3.9.4", "spatial-r1-v4.0.1", "spatial-r1-v4.1"])
def test_routing_diagnostics_from_the_gate_epilogue(cb, version):
    """On log steps the gate kernel accumulates the routing diagnostics itself; they must
    agree with the same statistics computed by the torch restatement of the op."""
    from dawn_srw_b200.ops.backend import ParallelCtx
    from dawn_srw_b200.ops.gates import gate_spec_for
    T, R, U, r, D = 300, 2, 1580, 64, 256
    dev = torch.device("cuda")
    torch.manual_seed(5)
    spec = gate_spec_for(version)
    be = cb.CudaBackend()
    nz = torch.nn.functional.normalize
    q = lambda t: t.bfloat16().float()
    emb, read, write = (q(nz(torch.randn(U, d, device=dev), dim=-1)) for d in (r, D, D))
    x, h = q(torch.randn(T, D, device=dev)), q(torch.randn(T, R, r, device=dev))
    off = torch.randn(T, R, device=dev) * 0.3 - 0.3
    with torch.no_grad():
        pool = be.prepare_pool(emb, read, write, spec, ParallelCtx())
        got = be.srw(x, h, off, pool, spec, pctx=ParallelCtx(), want_diag=True).diag
        want = be._srw_library(x, h, off, pool, spec, ParallelCtx(), True, False, None).diag
    cb.check_status()
    assert set(got) == set(want)
    loose = {"score_skew", "score_kurt", "gate_entropy"}     # higher moments / logs of bf16-level differences
    for k in want:
        a, b = got[k].float(), want[k].float()
        scale = float(b.abs().max()) + 1e-3
        err = float((a - b).abs().max()) / scale
        assert err < (0.1 if k in loose else 2e-2), (k, err, a.flatten()[:4], b.flatten()[:4])


def test_layernorm_kernel(cb):
    from dawn_srw_b200.ops import reference as R
    dev = torch.device("cuda")
    for T, D in ((300, 384), (129, 1280), (1, 1280), (5, 2048), (1500, 2048), (40, 4096)):
        x = (torch.randn(T, D, device=dev) * 3 + 1).requires_grad_(True)
        w = torch.randn(D, device=dev).requires_grad_(True)
        b = torch.randn(D, device=dev).requires_grad_(True)
        y = cb._LayerNormFn.apply(x, w, b)
        assert y.dtype == torch.bfloat16
        gy = torch.randn(T, D, device=dev).bfloat16()
        y.backward(gy)
        x2, w2, b2 = (t.detach().clone().requires_grad_(True) for t in (x, w, b))
        y2 = R.layer_norm(x2, w2, b2)
        y2.backward(gy.float())
        assert _rel(y, y2) < 4e-3
        assert _rel(x.grad, x2.grad) < 1e-4 and _rel(w.grad, w2.grad) < 1e-4 and _rel(b.grad, b2.grad) < 1e-4


def test_dropout_with_residual_add_and_regenerated_mask(cb):
    dev = torch.device("cuda")
    torch.manual_seed(5)
    be = cb.CudaBackend()
    res = torch.randn(512, 1280, device=dev)
    x = (torch.rand(512, 1280, device=dev) + 0.5).requires_grad_(True)      # no zeros: the mask is y != res
    p = 0.1
    y = be.dropout_add(res, x, p, True)
    kept = (y - res) != 0
    frac = kept.float().mean().item()
    assert abs(frac - (1 - p)) < 5e-3, frac
    assert torch.allclose((y - res)[kept], (x.detach() / (1 - p))[kept], rtol=1e-5, atol=1e-6)
    # rows and columns are not correlated: every column keeps about 90 %
    assert (kept.float().mean(0) - (1 - p)).abs().max() < 0.08
    gy = torch.randn_like(y)
    y.backward(gy)
    assert torch.allclose(x.grad, gy * kept / (1 - p), rtol=1e-5, atol=1e-6)   # same mask, regenerated
    # a second call draws another mask; evaluation is the identity
    y2 = be.dropout_add(res, x.detach(), p, True)
    assert ((y2 - res) != 0).ne(kept).any()
    assert torch.equal(be.dropout_add(res, x.detach(), p, False), res + x.detach())
    z = be.dropout(x.detach(), 0.25, True)
    assert abs((z != 0).float().mean().item() - 0.75) < 5e-3


def test_lm_head_cross_entropy(cb):
    from dawn_srw_b200.ops import reference as R
    dev = torch.device("cuda")
    be = cb.CudaBackend()
    B, S, D, V = 3, 40, 128, 1003
    x = torch.randn(B, S, D, device=dev).bfloat16().float().requires_grad_(True)
    emb = (torch.randn(V, D, device=dev) * 0.1).bfloat16().float().requires_grad_(True)
    labels = torch.randint(0, V, (B, S), device=dev)
    labels[0, 5:9] = -100
    loss, per_tok, correct, nvalid, vmask = be.lm_head_ce(x, emb, labels)
    loss.backward()
    x2, emb2 = x.detach().clone().requires_grad_(True), emb.detach().clone().requires_grad_(True)
    l2, pt2, c2, n2, _ = R.lm_head_ce(x2, emb2, labels)
    l2.backward()
    assert abs(float(loss) - float(l2)) < 2e-3 and int(nvalid) == int(n2) and int(correct) == int(c2)
    assert _rel(per_tok, pt2) < 2e-3
    assert _rel(x.grad, x2.grad) < 1e-2 and _rel(emb.grad, emb2.grad) < 1e-2


def test_kernels_are_run_to_run_deterministic(cb):
    """Every tile-produced output must be bit-identical between two runs (a
    missing barrier or a racing tile shows up here); only the per-token sums
    that are accumulated with atomics may differ in the last bits.  Products with
    few tiles and a long K, which are cut: test_split_products_repeat_bit_by_bit; row
    and column sums of the backward pass have tests of their own; not promised to
    repeat: denominators, LayerNorm's and the embeddings' gradients, and products
    that accumulate (pool gradients, Gram matrices, write GEMMs of generation)."""
    from dawn_srw_b200.ops.gates import GateSpec
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(9)
    T, U, r, D = 1024, 2504, 128, 384
    nz = torch.nn.functional.normalize
    rn = lambda *s: torch.randn(*s, device=dev, generator=g)
    h, x, dy = rn(T, r).bfloat16(), rn(T, D).bfloat16(), (rn(T, D) * 0.1).bfloat16()
    emb, read, write = (nz(rn(U, d), dim=-1).bfloat16() for d in (r, D, D))
    tau, isd, dden = torch.full((T,), 0.2, device=dev), torch.ones(T, device=dev), rn(T) * 0.01
    e, st, gl = cb.ext(), cb.status_word(dev), cb._gate_list(GateSpec(kind=1))
    runs = []
    for _ in range(2):
        p = torch.zeros(T, U, device=dev, dtype=torch.bfloat16)
        pb, dxr, ds = (torch.zeros_like(p) for _ in range(3))
        den, dtau, dsz = (torch.zeros(T, device=dev) for _ in range(3))
        e.srw_fwd_gate(h, emb, x, read, p, tau, isd, den, None, None, None, gl, st)
        y = cb.gemm(p, False, write, True, out_dtype=torch.float32)
        e.srw_bwd_gate(h, emb, x, read, dy, write, pb, dxr, ds, tau, isd, dden, dtau, dsz, gl, st)
        gw = cb.gemm(pb, True, dy, True, out_dtype=torch.float32)
        q = rn(2, 256, 4 * 64).bfloat16() if not runs else runs[0][-1]
        o = cb.causal_attention(q, q, q, 4, 0.1, 77)
        runs.append([p, y, pb, dxr, ds, gw, o, den, dtau, q])
    torch.cuda.synchronize()
    cb.check_status()
    for a, b in zip(runs[0][:7], runs[1][:7]):
        assert torch.equal(a, b)
    for a, b in zip(runs[0][7:9], runs[1][7:9]):
        assert torch.allclose(a, b, rtol=1e-5, atol=1e-5)


def _attn_ref(q, k, v, H, keep=None, p_drop=0.0):
    """fp32 dense causal attention on [B, S, H*dh]; ``keep`` is a [B,H,S,S] 0/1 mask."""
    B, S, D = q.shape
    dh = D // H
    hd = lambda t: t.float().view(B, S, H, dh).transpose(1, 2)
    s = hd(q) @ hd(k).transpose(-1, -2) / dh ** 0.5
    s = s.masked_fill(~torch.ones(S, S, dtype=torch.bool, device=q.device).tril(), float("-inf"))
    w = torch.softmax(s, -1)
    if keep is not None:
        w = w * keep / (1.0 - p_drop)
    return (w @ hd(v)).transpose(1, 2).reshape(B, S, D)


@pytest.mark.parametrize("shape", [(2, 4, 512, 80), (3, 2, 200, 64), (1, 3, 64, 32),
                                   (2, 2, 384, 128), (1, 1, 7, 16), (1, 2, 130, 96)])
def test_attention_kernels_against_fp32_reference(cb, shape):
    B, H, S, dh = shape
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(3)
    mk = lambda: (torch.randn(B, S, H * dh, device=dev, generator=g)).bfloat16().float().requires_grad_(True)
    q, k, v = mk(), mk(), mk()
    w = torch.randn(B, S, H * dh, device=dev, generator=g)
    out = cb.causal_attention(q, k, v, H)
    (out.float() * w).sum().backward()
    got = [out.float(), q.grad.clone(), k.grad.clone(), v.grad.clone()]
    q.grad = k.grad = v.grad = None
    ref = _attn_ref(q, k, v, H)
    (ref * w).sum().backward()
    want = [ref, q.grad, k.grad, v.grad]
    cb.check_status()
    for name, a, b in zip(("out", "dq", "dk", "dv"), got, want):
        assert _rel(a, b) < 1.5e-2, (name, _rel(a, b))


def test_attention_dropout_mask_is_shared_by_forward_and_backward(cb):
    """Recover the kernel's keep-mask with V = identity (S <= dh), then check
    forward and backward on random tensors against the reference with that mask."""
    B, H, S, dh, p_drop, seed = 2, 2, 128, 128, 0.25, 1234
    dev = torch.device("cuda")
    z = torch.zeros(B, S, H * dh, device=dev)
    eye = torch.eye(S, dh, device=dev).repeat(1, H).unsqueeze(0).repeat(B, 1, 1)
    o = cb.causal_attention(z, z, eye, H, p_drop, seed).float()
    keep = (o.view(B, S, H, dh).transpose(1, 2) > 0).float()          # [B,H,S,S]
    tri = torch.ones(S, S, device=dev).tril()
    frac = float((keep * tri).sum() / (tri.sum() * B * H))
    assert abs(frac - (1 - p_drop)) < 0.02, frac
    g = torch.Generator(device=dev).manual_seed(5)
    mk = lambda: torch.randn(B, S, H * dh, device=dev, generator=g).bfloat16().float().requires_grad_(True)
    q, k, v = mk(), mk(), mk()
    w = torch.randn(B, S, H * dh, device=dev, generator=g)
    out = cb.causal_attention(q, k, v, H, p_drop, seed)
    (out.float() * w).sum().backward()
    got = [out.float(), q.grad.clone(), k.grad.clone(), v.grad.clone()]
    q.grad = k.grad = v.grad = None
    ref = _attn_ref(q, k, v, H, keep, p_drop)
    (ref * w).sum().backward()
    cb.check_status()
    for name, a, b in zip(("out", "dq", "dk", "dv"), got, [ref, q.grad, k.grad, v.grad]):
        assert _rel(a, b) < 1.5e-2, (name, _rel(a, b))


def test_embedding_kernels(cb):
    from dawn_srw_b200.ops import reference as R
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(0)
    V, P, D, B, S = 300, 40, 132, 5, 33
    tok = torch.randn(V, D, device=dev, generator=g, requires_grad=True)
    pos = torch.randn(P, D, device=dev, generator=g, requires_grad=True)
    ids = torch.randint(0, V, (B, S), device=dev, generator=g)
    ids[0, :5] = 7                                            # repeated tokens collide in backward
    w = torch.randn(B, S, D, device=dev, generator=g)
    be = cb.CudaBackend()
    out = be.embed(ids, tok, pos)
    (out * w).sum().backward()
    got = [out.detach(), tok.grad.clone(), pos.grad.clone()]
    tok.grad = pos.grad = None
    ref = R.embed(ids, tok, pos)
    (ref * w).sum().backward()
    assert torch.equal(got[0], ref.detach())
    assert torch.allclose(got[1], tok.grad, atol=1e-5) and torch.allclose(got[2], pos.grad, atol=1e-5)


def test_diversity_kernel_and_padded_heads(cb):
    from dawn_srw_b200.ops import reference as R
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(1)
    ws = [torch.randn(n, d, device=dev, generator=g, requires_grad=True)
          for n, d in ((520, 64), (9000, 128), (300, 72))]
    be = cb.CudaBackend()
    val = be.diversity(ws)
    val.backward()
    got = [w.grad.clone() for w in ws]
    for w in ws:
        w.grad = None
    ref = R.pool_diversity(ws)
    ref.backward()
    assert abs(float(val) - float(ref)) < 2e-3 * float(ref)
    for a, w in zip(got, ws):
        assert _rel(a, w.grad) < 0.08, _rel(a, w.grad)        # bf16 rounding flips the sign of near-zero cosines
    # a 3-wide head (tau projection) runs on the engine through zero padding
    x = torch.randn(300, 128, device=dev, generator=g, requires_grad=True)
    w3 = torch.randn(3, 128, device=dev, generator=g, requires_grad=True)
    b3 = torch.randn(3, device=dev, generator=g, requires_grad=True)
    y = be.linear(x, w3, b3)
    y.square().sum().backward()
    gy = [x.grad.clone(), w3.grad.clone(), b3.grad.clone()]
    x.grad = w3.grad = b3.grad = None
    yr = torch.nn.functional.linear(x, w3, b3)
    yr.square().sum().backward()
    assert y.shape == (300, 3) and _rel(y, yr) < 1e-2
    for a, b_ in zip(gy, (x.grad, w3.grad, b3.grad)):
        assert _rel(a, b_) < 2e-2
    cb.check_status()


def test_fused_adamw_and_grad_norm(cb):
    from dawn_srw_b200.train.optimizer import DawnAdamW
    dev = torch.device("cuda")
    torch.manual_seed(0)
    shapes = [(130, 70), (70,), (1000, 33), (300, 701), (3,)]      # one tensor spans several 64 K chunks
    names = ["router.proj_know.weight", "router.proj_know.bias", "neuron_pool.know_read",
             "layers.0.attn.expand_O.weight", "router.tau_attn.bias"]
    pa = [torch.nn.Parameter(torch.randn(*s, device=dev)) for s in shapes]
    pb = [torch.nn.Parameter(p.detach().clone()) for p in pa]
    oa = DawnAdamW(list(zip(names, pa)), lr=1e-2, fused=True)
    ob = DawnAdamW(list(zip(names, pb)), lr=1e-2, fused=False)
    for _ in range(3):
        gs = [torch.randn(*s, device=dev) * 2 for s in shapes]
        for p, q, g in zip(pa, pb, gs):
            p.grad, q.grad = g.clone(), g.clone()
        oa.step(), ob.step()
    assert abs(float(oa.last_grad_norm) - float(ob.last_grad_norm)) < 1e-3
    for p, q in zip(pa, pb):
        assert torch.allclose(p, q, atol=2e-6)
    # the backend's cached bf16 compute copy follows a weight the kernel rewrote
    be = cb.CudaBackend()
    w0 = be._w(pa[0]).clone()
    pa[0].grad = torch.ones_like(pa[0])
    oa.step()
    assert not torch.equal(be._w(pa[0]), w0)
    assert torch.equal(be._w(pa[0]), pa[0].detach().to(torch.bfloat16))


def test_tiny_model_matches_reference_backend_and_trains(cb):
    from dawn_srw_b200.models.dawn import DAWN
    from dawn_srw_b200.ops.backend import ReferenceBackend
    dev = torch.device("cuda")
    kw = dict(vocab_size=1000, d_model=128, n_layers=2, n_heads=4, max_seq_len=64, d_route=64,
              n_qk=200, n_v=264, n_know=520, model_version="spatial-r1-v4.0.1", dropout_rate=0.0,
              router_dropout=0.0)
    m1 = DAWN(**kw, backend=ReferenceBackend(torch.float32)).to(dev)
    m2 = DAWN(**kw, backend=cb.CudaBackend()).to(dev)
    m2.load_state_dict(m1.state_dict())
    ids = torch.randint(0, 1000, (4, 64), device=dev, generator=torch.Generator(device=dev).manual_seed(7))
    outs = []
    for m in (m1, m2):
        r = m(ids, labels=ids, want_diag=False)
        (r["loss"] + 0.1 * r["aux_loss"]).backward()
        outs.append(r)
    assert abs(float(outs[0]["loss"]) - float(outs[1]["loss"])) < 5e-3
    assert abs(float(outs[0]["aux_loss"]) - float(outs[1]["aux_loss"])) < 5e-3
    for (n, p1), (_, p2) in zip(m1.named_parameters(), m2.named_parameters()):
        if p1.grad is not None and p1.grad.abs().max() > 0 and p1.numel() > 4:
            # (tiny tensors such as the tau biases are sums with heavy cancellation)
            assert _rel(p2.grad, p1.grad) < 0.08, (n, _rel(p2.grad, p1.grad))
    # diagnostics path on the CUDA backend
    r = m2(ids, labels=ids, want_diag=True)
    assert "know_active" in r and 0.0 <= float(r["know_active"]) <= 1.0
    cb.check_status()


def test_graph_captured_decoding_matches_eager_and_prefill(cb):
    """The per-token step replayed from a CUDA graph gives the logits of the eager step,
    and both agree with a full-sequence forward over the same tokens."""
    from dawn_srw_b200.models import inference as I
    from dawn_srw_b200.models.dawn import DAWN
    dev = torch.device("cuda")
    m = DAWN(vocab_size=1000, d_model=128, n_layers=2, n_heads=4, max_seq_len=64, d_route=64, n_qk=200,
             n_v=264, n_know=1100, model_version="spatial-r1-v4.0.1", dropout_rate=0.0,
             router_dropout=0.0, backend=cb.CudaBackend()).to(dev).eval()
    g = torch.Generator(device=dev).manual_seed(3)
    ids = torch.randint(1, 1000, (3, 12), device=dev, generator=g)
    more = torch.randint(1, 1000, (3, 5), device=dev, generator=g)
    logits_p, ck, cv, n = I.prefill(m, ids)
    sess_g = I.DecodeSession(m, ck.clone(), cv.clone(), n, use_graph=True)
    sess_e = I.DecodeSession(m, ck.clone(), cv.clone(), n, use_graph=False)
    got_g, got_e = [], []
    for t in range(more.shape[1]):
        got_g.append(sess_g.step(more[:, t]))
        got_e.append(sess_e.step(more[:, t]))
    assert sess_g.graph is not None and sess_g.length == n + more.shape[1]
    full = I.prefill(m, torch.cat([ids, more], dim=1))[0]          # [B, S, V]
    for t in range(more.shape[1]):
        assert _rel(got_g[t], got_e[t]) < 1e-3
        assert _rel(got_g[t], full[:, n + t]) < 2e-2
    out_g, _ = I.generate(m, ids, max_new_tokens=6, temperature=0.0, use_graph=True)
    out_e, _ = I.generate(m, ids, max_new_tokens=6, temperature=0.0, use_graph=False)
    assert torch.equal(out_g, out_e)
    cb.check_status()


def test_training_reduces_loss_on_gpu(cb):
    from dawn_srw_b200.config import preset
    from dawn_srw_b200.train.trainer import Trainer
    cfg = preset("400M", d_model=128, n_layers=2, n_heads=4, d_route=64, n_qk=200, n_v=264, n_know=1000)
    cfg.model.vocab_size, cfg.model.max_seq_len = 512, 64
    cfg.model.dropout = cfg.model.router_dropout = 0.0
    cfg.training.batch_size, cfg.training.lr = 8, 3e-3
    cfg.data.synthetic = True
    tr = Trainer(cfg, device=torch.device("cuda", 0), total_steps=1000)
    assert tr.backend.name == "sm100a"
    ids, mask = tr.train_loader.batch(0)
    first = float(tr.train_step(ids, mask)["ce_loss"])
    for _ in range(40):
        last = float(tr.train_step(ids, mask)["ce_loss"])
    assert last < first - 0.5
    assert cb.launch_count() > 0


def test_graft_entry_smoke():
    import __graft_entry__ as g
    g.smoke()


@pytest.mark.parametrize("U,r,layers", [(1, 8, 1), (7, 16, 2), (130, 128, 3), (1001, 256, 30), (2600, 384, 2),
                                        (77, 512, 25)])
def test_load_balance_term_and_its_gradients(cb, U, r, layers):
    """One lane to a warp per unit, one or two chunks per lane, more layers than one launch of the
    outer products takes.  fp32 sums of up to U terms against fp64: 1e-5 covers sqrt(U) roundings;
    var is a difference of nearly equal numbers only where the mean dominates, which it does not."""
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(U + r)
    rn = lambda *s: torch.randn(*s, device=dev, generator=g)
    hd = cb._PoolTensors()
    hd.emb = rn(U + 3, r).bfloat16()
    hd.g_emb = rn(U + 3, r)
    ref_e = hd.emb[:U].double().requires_grad_(True)
    start = hd.g_emb.clone()
    total = 0.0
    for k in range(layers):
        hsum = (rn(r) * 40).requires_grad_(True)
        lb = cb._LoadBalanceFn.apply(hsum, torch.zeros(1, device=dev), hd, U, 1.0 / 96, float(U))
        (lb * (k + 1.5)).backward()
        hs = hsum.detach().double().requires_grad_(True)
        m = ref_e @ (hs / 96)
        mean = m.sum() / U
        var = (m * m).sum() / U - mean ** 2
        ref = var / (mean ** 2 + var + 1e-2)
        (ref * (k + 1.5)).backward()
        assert abs(float(lb) - float(ref)) < 1e-5
        assert float((hsum.grad.double() - hs.grad).norm()) < 1e-4 * float(hs.grad.norm()) + 1e-6
    pairs, hd.rank1 = hd.rank1, []
    cb.ext().rank1_add(hd.g_emb[:U], torch.stack([d for d, _ in pairs]), torch.stack([h for _, h in pairs]))
    added = (hd.g_emb - start).double()
    assert float(added[U:].abs().max()) == 0.0
    # every layer's product is added to a value of order one: 2^-24 of rounding per element each
    rounding = 2.0 ** -24 * (layers * U * r) ** 0.5
    assert float((added[:U] - ref_e.grad).norm()) < 1e-4 * float(ref_e.grad.norm()) + rounding + 1e-6


@pytest.mark.parametrize("T,R,r,wide", [(1, 1, 8, 24), (5, 2, 16, 35), (129, 2, 64, 131), (300, 1, 384, 387)])
def test_stacked_call_statistics_and_row_steps(cb, T, R, r, wide):
    """Routes that are strided (and here unaligned) slices of a router output, stacked for one
    call: bf16 copy exact, statistics and their gradients against fp64 of the same bf16 values;
    2e-5 covers the two-term Gram split (2^-17), 3e-3 gradients through bf16(d_var h)."""
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(T + r)
    rn = lambda *s: torch.randn(*s, device=dev, generator=g)
    U, e, st = 600, cb.ext(), cb.status_word(dev)
    h = rn(T, R * r + wide)[:, 3:3 + R * r].unflatten(1, (R, r))
    off = (rn(T, R + 2) * 0.3)[:, 1:1 + R]
    emb = torch.nn.functional.normalize(rn(U, r), dim=-1).bfloat16().double()
    gram, esum = emb.t() @ emb, emb.sum(0)
    hi = gram.float().bfloat16()
    gcat = torch.cat([hi, (gram.float() - hi.float()).bfloat16()])
    hb, hg, tau, isd, mu, sd, den, hsum = e.srw_stats(h, off, gcat, esum.float(), 1.0 / U, st)
    assert torch.equal(hb.view(R, T, r), h.transpose(0, 1).bfloat16())
    assert float(den.abs().max()) == 0.0
    h64, o64 = hb.double().requires_grad_(True), off.t().reshape(-1).double().requires_grad_(True)
    gr64, es64 = gram.clone().requires_grad_(True), esum.clone().requires_grad_(True)
    m = (h64 @ es64) / U
    s = (((h64 @ gr64) * h64).sum(-1) / U - m * m).sqrt()
    t64 = m + o64 * s
    assert _rel(tau, t64) < 2e-5 and _rel(isd, 1 / s) < 2e-5 and _rel(hsum, h64.sum(0)) < 1e-5
    dtau, dh32, d_hsum = rn(R * T), rn(R * T, r), rn(r)
    d_isd = (((hb.double() * dh32.double()).sum(-1) + t64.detach() * dtau) * s.detach())     # dsz / isd^2
    ((t64 * dtau).sum() + (d_isd / s).sum() + (h64 * (dh32 + d_hsum).double()).sum()).backward()
    g_gram, g_esum = torch.zeros(r, r, device=dev), torch.zeros(r, device=dev)
    dh, d_off = e.srw_stats_bwd(dtau, dh32, d_hsum, off, tau, isd, mu, sd, hg, hb, esum.float(), 1.0 / U,
                                True, g_gram, g_esum, st)
    cb.check_status()
    assert _rel(dh.transpose(0, 1).reshape(R * T, r), h64.grad) < 1e-4
    assert _rel(d_off.t().reshape(-1), o64.grad) < 1e-4 and _rel(g_esum, es64.grad) < 1e-4
    assert _rel(g_gram + g_gram.t(), gr64.grad + gr64.grad.t()) < 2 * 3e-3


@pytest.mark.parametrize("T,D", [(1, 8), (9, 136), (64, 2048)])
def test_route_backward_row_step(cb, T, D):
    """Denominators below, at and above one, and NaN (which has to reach the operand, as with
    clamp); fp32 sums of D terms, so 1e-5, and one bf16 rounding of the operand."""
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(T)
    rn = lambda *s: torch.randn(*s, device=dev, generator=g)
    dy, y, den = rn(T, D), rn(T, D), rn(T).abs() * 2
    den[0] = 1.0
    scale, ext_dden = torch.full((), 1.7, device=dev), rn(T)
    dtau, d_scale = rn(T), torch.zeros((), device=dev)
    dyb, d_den = cb.ext().route_bwd_rows(dy, y, den, 1.0, scale, ext_dden, dtau, d_scale)
    dot = (dy.double() * y.double()).sum(-1)
    assert torch.equal(dyb, (dy * (scale / den.clamp(min=1.0))[:, None]).bfloat16()) or \
        _rel(dyb, dy * (scale / den.clamp(min=1.0))[:, None]) < 4e-3
    want = torch.where(den > 1.0, -dot / den, torch.zeros_like(dot)) + ext_dden
    assert float((d_den - want).abs().max()) < 1e-5 * D and float(dtau.abs().max()) == 0.0
    assert abs(float(d_scale) - float(dot.sum() / 1.7)) < 1e-5 * T * D
    den[0] = float("nan")
    dyb, _ = cb.ext().route_bwd_rows(dy, y, den, 1.5, None, None, dtau, None)
    assert bool(dyb[0].isnan().all()) and bool(dyb[1:].isfinite().all())


@pytest.mark.parametrize("T,R,r", [(1, 1, 8), (2, 2, 120), (1, 2, 136), (64, 2, 384), (5, 1, 512)])
def test_score_statistics_of_a_few_rows_over_a_cluster(cb, T, R, r):
    """CTAs with no row of G, with fewer and with more than sixteen; strided inputs; the scratch
    that the launch clears.  fp32 sums of r^2 terms against fp64: 2e-5."""
    from dawn_srw_b200.ops.score_stats import score_stats_rows
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(r)
    rn = lambda *s: torch.randn(*s, device=dev, generator=g)
    h, off = rn(T, R * r + 5)[:, 2:2 + R * r].unflatten(1, (R, r)), rn(T, R + 1)[:, :R]
    emb = rn(700, r).double() / r ** 0.5
    gram, esum = emb.t() @ emb, emb.sum(0)
    tau, isd, hb, zero = score_stats_rows(h, off, gram.float(), esum.float(), 700, 10007)
    assert torch.equal(hb, h.transpose(0, 1).reshape(R * T, r).bfloat16())
    assert zero.numel() == 10007 and float(zero.abs().max()) == 0.0
    hd = hb.double()
    mu = hd @ esum / 700
    sd = (((hd @ gram) * hd).sum(-1) / 700 - mu * mu).sqrt()
    assert _rel(tau, mu + off.t().reshape(-1).double() * sd) < 2e-5 and _rel(isd, 1 / sd) < 2e-5


@pytest.mark.parametrize("N,x_rows,U,D,r", [(1, 1, 1, 8, 8), (2, 1, 300, 128, 16), (4, 2, 2999, 256, 264),
                                            (2, 2, 160000, 64, 8), (1, 1, 6400, 2048, 512)])
def test_streaming_pool_op_over_unit_counts(cb, N, x_rows, U, D, r):
    """Blocks without a unit, lanes shared by several units, more units per block than its list
    holds, rows that share an x row, a mask; against the formula with p rounded to bf16 (3e-3)."""
    from dawn_srw_b200.ops.gates import GateSpec, gate_forward
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(U)
    rn = lambda *s: torch.randn(*s, device=dev, generator=g)
    spec = GateSpec(kind=1)
    h, x = rn(N, r).bfloat16(), rn(x_rows, D).bfloat16()
    emb, read, write = rn(U, r).bfloat16(), rn(U, D).bfloat16(), rn(U, D).bfloat16()
    mask = (torch.rand(U, device=dev, generator=g) < 0.8).float()
    s = h.float() @ emb.float().t()
    sd = s.std(-1, unbiased=False, keepdim=True) + 1.0
    tau = s.mean(-1, keepdim=True) - 0.1
    gate, dt, _ = gate_forward(spec, s, tau, sd)
    xn = x.repeat(N // x_rows, 1).float()
    p = (gate * mask * (xn @ read.float().t())).bfloat16().float()
    ref = (p @ write.float()) * (0.7 / (dt * mask).sum(-1).clamp(min=1.0))[:, None]
    first = None
    for _ in range(3):
        out, den = cb.ext().srw_rows(h, x, tau.squeeze(-1).contiguous(), (1 / sd).squeeze(-1).contiguous(),
                                     emb, read, write, mask, cb._gate_list(spec), 0.7, None)
        assert _rel(out, ref) < 3e-3 and _rel(den, (dt * mask).sum(-1)) < 1e-4
        first = out if first is None else first
        assert torch.equal(out, first)                       # every sum has a fixed order


@pytest.mark.parametrize("kind", [0, 1, 2])
@pytest.mark.parametrize("T,U,D,r", [(5, 520, 136, 64), (16, 1000, 384, 128), (17, 5003, 256, 72),
                                     (33, 16100, 2048, 384), (64, 1580, 1280, 256), (65, 700, 128, 64)])
def test_route_of_a_few_rows_on_the_tensor_engine(cb, kind, T, U, D, r):
    """Token tiles of 16, 32 and 64 with ragged rows, units and columns, a mask, K cut into splits,
    and one row too many for the swapped form; the formula with p rounded to bf16, so 6e-3."""
    from dawn_srw_b200.ops.gates import GateSpec, gate_forward
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(U + kind)
    rn = lambda *s: torch.randn(*s, device=dev, generator=g)
    spec, Up = GateSpec(kind=kind), (U + 7) // 8 * 8
    nz = lambda *s: torch.nn.functional.normalize(rn(*s), dim=-1).bfloat16()
    h, x, emb, read, write = rn(T, r).bfloat16(), rn(T, D).bfloat16(), nz(U, r), nz(U, D), nz(U, D)
    mask = (torch.rand(U, device=dev, generator=g) < 0.9).float()
    s = h.float() @ emb.float().t()
    sd = s.std(-1, unbiased=False, keepdim=True)
    tau = s.mean(-1, keepdim=True) + 0.6 * sd
    gate, dt, _ = gate_forward(spec, s, tau, sd)
    p_ref = (gate * mask * (x.float() @ read.float().t())).bfloat16().float()
    ref = (p_ref @ write.float()) * (1.3 / (dt * mask).sum(-1).clamp(min=1.0))[:, None]
    st, scale = cb.status_word(dev), torch.full((1,), 1.3, device=dev)
    for sc_f, sc_t in ((1.3, None), (1.0, scale)):
        p = torch.empty(T, Up, device=dev, dtype=torch.bfloat16)
        y, den = torch.zeros(T, D, device=dev), torch.zeros(T, device=dev)
        cb.ext().srw_route_fwd(h, x, emb, read, write, p, None, tau.squeeze(-1).contiguous(),
                               (1 / sd).squeeze(-1).contiguous(), den, None, None, mask,
                               cb._gate_list(spec), sc_f, sc_t, y, True, st)
        cb.check_status()
        assert _rel(den, (dt * mask).sum(-1)) < 1e-4
        assert _rel(p[:, :U], p_ref) < 8e-3 and _rel(y, ref) < 6e-3


@pytest.mark.parametrize("M", [5, 16, 31, 64])
def test_gemm_of_a_few_rows_with_swapped_operands(cb, M):
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(M)
    for K, N in ((64, 8), (200, 131), (2048, 1283)):
        Kp = (K + 7) // 8 * 8
        x = torch.randn(M, Kp, device=dev, generator=g).bfloat16()[:, :K]
        w = torch.randn(N, Kp, device=dev, generator=g).bfloat16()[:, :K]
        bias = torch.randn(N, device=dev, generator=g)
        ref = 0.5 * (x.double() @ w.double().t()) + bias
        out = cb.gemm(x, False, w, False, out_dtype=torch.float32, bias=bias, alpha=0.5)
        assert out.shape == (M, N) and _rel(out, ref) < 1e-5
    cb.check_status()


@pytest.mark.parametrize("M,N,K,a_mn", [(384, 384, 8192, True), (8, 384, 8200, True), (512, 384, 25200, False),
                                        (300, 131, 10400, False), (256, 128, 4096, True)])
def test_plain_gemm_with_few_tiles_and_a_long_k(cb, M, N, K, a_mn):
    """K is cut although the caller does not accumulate: whatever the output held is gone, rows
    beyond its width stay, and the row scale applies to the sum of the parts (fp32 sums: 1e-5)."""
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(K + M)
    A = torch.randn(M, K, device=dev, generator=g).bfloat16()
    B = torch.randn((N + 7) // 8 * 8, K, device=dev, generator=g).bfloat16()[:N]
    rs = torch.rand(M, device=dev, generator=g)
    buf = torch.full((M, (N + 7) // 8 * 8 + 8), float("nan"), device=dev)
    ref = 0.3 * (A.double() @ B.double().t()) * rs[:, None]
    cb.gemm(A.t().contiguous() if a_mn else A, a_mn, B, False, out=buf[:, :N], alpha=0.3, row_scale=rs)
    cb.check_status()
    assert _rel(buf[:, :N], ref) < 1e-5 and bool(buf[:, N:].isnan().all())


@pytest.mark.parametrize("T,D,n1,n2,p", [(1, 64, 8, 1, 0.0), (65, 136, 24, 3, 0.0), (300, 384, 384, 3, 0.1),
                                         (257, 128, 128, 1, 0.1)])
def test_router_projection_and_its_gradients(cb, T, D, n1, n2, p):
    """One GEMM for projection and thresholds: pieces, ragged column cuts, dropout and the packed
    backward operand (cotangents of overlapping thresholds add up) against the separate layers;
    bf16 operands on both sides, so 1e-2 on gradients."""
    dev = torch.device("cuda")
    torch.manual_seed(T)
    be = cb.CudaBackend()
    proj, tau = torch.nn.Linear(D, n1).to(dev), torch.nn.Linear(D, n2).to(dev)
    x0 = torch.randn(T, D, device=dev)
    cuts, tcuts = ((n1 // 3 * 2, n1 - n1 // 3 * 2), (n2 - 1, 1)) if n2 > 1 else ((n1,), (1,))
    wh, wt, wa = torch.randn(T, n1, device=dev), torch.randn(T, n2, device=dev), torch.randn(T, n2, device=dev)
    got = []
    for fused in (True, False):
        for l in (proj, tau):
            l.zero_grad()
        x = x0.clone().requires_grad_(True)
        torch.manual_seed(7)
        if fused:
            hs, ts, ta = be.router(x, proj, tau, p, True, cuts, tcuts)
            h, t = torch.cat(hs, 1), torch.cat(ts, 1)
        else:
            h = be.dropout(be.linear(x, proj.weight, proj.bias).contiguous(), p, True)
            t = ta = be.linear(x, tau.weight, tau.bias)
        ((h * wh).sum() + (t * wt).sum() + (ta * wa).sum()).backward()
        got.append([h.detach(), t.detach(), ta.detach(), x.grad] + [q.grad.clone() for l in (proj, tau)
                                                                    for q in (l.weight, l.bias)])
    cb.check_status()
    for a, b in zip(*got):
        assert _rel(a, b) < 1e-2
    ref = torch.nn.functional.linear(x0.double(), proj.weight.double(), proj.bias.double())
    kept = got[0][0] != 0
    assert _rel(got[0][0][kept] * (1 - p), ref[kept]) < 1e-2


@pytest.mark.parametrize("B,S,H,dh,s_max", [(1, 1, 1, 16, 1), (3, 109, 6, 64, 128), (2, 130, 2, 80, 131),
                                            (1, 257, 3, 128, 300)])
def test_prompt_attention_fills_the_caches(cb, B, S, H, dh, s_max):
    """Caches exact at 0..S-1 and untouched beyond; output as the attention entry point gives it."""
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(S)
    q, k, v = (torch.randn(B * S, H * dh, device=dev, generator=g) for _ in range(3))
    ck, cv = torch.full((2, B, H, s_max, dh), 7.0, device=dev).unbind(0)
    be = cb.CudaBackend()
    o = be.prompt_attention(q, k, v, ck, cv, B, S)
    heads = lambda t: t.view(B, S, H, dh).transpose(1, 2)
    assert torch.equal(ck[:, :, :S], heads(k)) and torch.equal(cv[:, :, :S], heads(v))
    assert bool((ck[:, :, S:] == 7.0).all()) and bool((cv[:, :, S:] == 7.0).all())
    ref = be.attention(heads(q), heads(k), heads(v), 0.0, False).transpose(1, 2).reshape(B * S, H * dh)
    cb.check_status()
    assert torch.equal(o, ref)


@pytest.mark.parametrize("T,D", [(297, 4), (300, 384), (513, 512), (1000, 516), (299, 1280), (320, 2048),
                                 (301, 130), (300, 2052)])
def test_layer_norm_over_row_lengths(cb, T, D):
    """Vector rows at the edges of their register tiles, a row length that is no multiple of four,
    one beyond the vector kernels; bf16 output and incoming gradient, so 8e-3 against fp64."""
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(D)
    rn = lambda *s: torch.randn(*s, device=dev, generator=g)
    x, w, b = (rn(T, D) * 2 + 1).requires_grad_(True), rn(D).requires_grad_(True), rn(D).requires_grad_(True)
    y = cb.CudaBackend().layer_norm(x, w, b)
    dy = rn(T, D).bfloat16()
    y.backward(dy)
    x6, w6, b6 = (t.detach().double().requires_grad_(True) for t in (x, w, b))
    ref = torch.nn.functional.layer_norm(x6, (D,), w6, b6, 1e-6)
    ref.backward(dy.double())
    assert _rel(y, ref) < 8e-3
    for a, r in ((x.grad, x6.grad), (w.grad, w6.grad), (b.grad, b6.grad)):
        assert _rel(a, r) < 1e-4


def test_decode_attention_with_scores_of_minus_infinity(cb):
    """A cached key whose score is -inf gets no weight wherever it falls: first of its group, alone
    in its group, or after others."""
    from dawn_srw_b200.ops import reference as R
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(3)
    B, H, dh, S, n = 2, 3, 64, 300, 200
    ck, cv = (torch.randn(B, H, S, dh, device=dev, generator=g) for _ in range(2))
    ck[:, :, [0, 1, 33, 64, 190], 5] = float("-inf")
    q = torch.rand(B, H * dh, device=dev, generator=g) + 0.1
    k, v = (torch.randn(B, H * dh, device=dev, generator=g) for _ in range(2))
    out = cb.CudaBackend().decode_attention(q, k, v, ck, cv, torch.tensor([n], device=dev), H)
    ref = R.cached_attention(q.view(B, H, 1, dh), ck, cv, n + 1).reshape(B, H * dh)
    assert bool(ref.isfinite().all()) and _rel(out, ref) < 1e-5


@pytest.mark.parametrize("sizes", [(1, 3, 4, 7), (1023, 1024, 1030), (65536, 65537, 200003)])
def test_multi_tensor_optimizer_over_sizes_and_alignments(cb, sizes):
    """Remainders of four, chunk edges, and tensors that start 4 bytes off a 16-byte boundary (the
    scalar form); one fp32 update, so 1e-6, and an fp32 sum of squares, so 1e-5."""
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(len(sizes))
    mk = lambda n, off: torch.randn(n + off, device=dev, generator=g)[off:]
    ts = [[mk(n, k % 2) for k, n in enumerate(sizes)] for _ in range(4)]
    p, gr, m, v = ts[0], ts[1], ts[2], [t.abs() for t in ts[3]]
    v = [mk(t.numel(), k % 2).abs_() for k, t in enumerate(v)]
    old = [[t.double().clone() for t in lst] for lst in (p, gr, m, v)]
    cs = torch.full((1,), 0.37, device=dev)
    total = cb.ext().grad_sq_norm(gr)
    cb.ext().adamw_multi(p, gr, m, v, cs, 1e-2, 0.9, 0.95, 1e-8, 0.1, 0.5, 0.3)
    assert _rel(total.reshape(()), sum((t * t).sum() for t in old[1])) < 1e-5
    for k in range(len(sizes)):
        po, go, mo, vo = (o[k] for o in old)
        go = go * 0.37
        mo, vo = 0.9 * mo + 0.1 * go, 0.95 * vo + 0.05 * go * go
        po = po - 1e-2 * ((mo / 0.5) / ((vo / 0.3).sqrt() + 1e-8) + 0.1 * po)
        for a, b in ((p[k], po), (m[k], mo), (v[k], vo)):
            assert _rel(a, b) < 1e-6


@pytest.mark.parametrize("D,n1,n2", [(64, 24, 3), (128, 128, 1), (2048, 1152, 3)])
def test_router_sees_every_write_to_its_parameters(cb, D, n1, n2):
    """Writes through .data move no version counter; the next call has to use them all the same.
    Against fp64 of the parameters as they are: bf16 operands, 1e-2."""
    dev = torch.device("cuda")
    torch.manual_seed(D)
    be, x = cb.CudaBackend(), torch.randn(70, D, device=dev)
    proj, tau = torch.nn.Linear(D, n1).to(dev), torch.nn.Linear(D, n2).to(dev)
    for q in (None, tau.bias, proj.bias, tau.weight, proj.weight):
        if q is not None:
            q.data.copy_(torch.randn_like(q))
        (h,), _, t = be.router(x, proj, tau, 0.0, False, (n1,), (n2,))
        for got, l in ((h, proj), (t, tau)):
            want = torch.nn.functional.linear(x.double(), l.weight.double(), l.bias.double())
            assert _rel(got, want) < 1e-2
    cb.check_status()


@pytest.mark.parametrize("n1,n2,D", [(8, 1, 4), (24, 3, 130), (768, 3, 1280), (5, 3, 64)])
def test_router_operand_rows(cb, n1, n2, D):
    dev = torch.device("cuda")
    w1, w2 = torch.randn(n1, D, device=dev), torch.randn(n2 * D + 1, device=dev)[1:].view(n2, D)   # 4 bytes off
    b1, b2 = torch.randn(n1, device=dev), torch.randn(n2, device=dev)
    for second in (w2, w2.clone()):
        w, b = cb.ext().router_operand(w1, b1, second, b2)
        n = (n1 + n2 + 7) // 8 * 8
        want = torch.zeros(n, D, device=dev)
        want[:n1], want[n1:n1 + n2] = w1, w2
        assert torch.equal(w, want.bfloat16())
        assert torch.equal(b, torch.nn.functional.pad(torch.cat([b1, b2]), (0, n - n1 - n2)))


@pytest.mark.parametrize("n2", [1, 3])
@pytest.mark.parametrize("bias", [True, False])
def test_router_takes_transposed_uses_and_layers_without_bias(cb, n2, bias):
    """A loss on the transposed thresholds gives a [T, 1] cotangent of strides (1, T), which counts as
    contiguous; bf16 operands on both sides, so 1e-2 against the separate layers in fp64."""
    dev = torch.device("cuda")
    torch.manual_seed(n2)
    be, T, D, n1 = cb.CudaBackend(), 69, 64, 24
    proj, tau = (torch.nn.Linear(D, n, bias=bias).to(dev) for n in (n1, n2))
    x = torch.randn(T, D, device=dev)
    wt, wh = torch.randn(n2, T, device=dev), torch.randn(n1, T, device=dev)
    xs = x.clone().requires_grad_(True)
    (h,), _, t = be.router(xs, proj, tau, 0.0, True, (n1,), (n2,))
    ((t.t() * wt).sum() + (h.t() * wh).sum()).backward()
    cb.check_status()
    want = [wt.t().double() @ tau.weight.double() + wh.t().double() @ proj.weight.double(),
            wt.double() @ x.double(), wh.double() @ x.double()]
    for a, b in zip((xs.grad, tau.weight.grad, proj.weight.grad), want):
        assert _rel(a, b) < 1e-2
    if bias:
        assert _rel(tau.bias.grad, wt.sum(1)) < 1e-2 and _rel(proj.bias.grad, wh.sum(1)) < 1e-2


@pytest.mark.parametrize("M,N,K,a_mn", [(512, 384, 25200, False), (384, 384, 8192, True), (300, 131, 10400, False),
                                        (8, 384, 8200, True), (129, 1280, 100000, False)])
def test_split_products_repeat_bit_by_bit(cb, M, N, K, a_mn):
    """A product that does not accumulate has the same bits in every run, also where K is cut: between
    the runs another product of other sizes moves the splits to other SMs and stale accumulators."""
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(M)
    A, B = torch.randn(M, K, device=dev, generator=g).bfloat16(), torch.randn(K, (N + 7) // 8 * 8, device=dev,
                                                                             generator=g).bfloat16()[:, :N]
    As = A.t().contiguous() if a_mn and M % 8 == 0 else A
    big = torch.randn(777, 1024, device=dev, generator=g).bfloat16()
    outs = []
    for k in range(6):
        cb.gemm(big[:100 * k + 1], False, big, False)
        outs.append(cb.gemm(As, As is not A, B, True, out_dtype=torch.float32))
    cb.check_status()
    assert _rel(outs[0], A.double() @ B.double()) < 1e-5
    assert all(torch.equal(outs[0], o) for o in outs[1:])


def test_route_backward_of_few_tokens_repeats_bit_by_bit(cb):
    """dx (in fp32, both routes added) and dh of a route against 25 200 units."""
    from dawn_srw_b200.ops.gates import GateSpec
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(1)
    rn = lambda *s: torch.randn(*s, device=dev, generator=g)
    nz = lambda *s: torch.nn.functional.normalize(rn(*s), dim=-1).bfloat16()
    T, U, r, D = 200, 25200, 128, 384
    h, x, dy, emb, read, write = rn(T, r).bfloat16(), rn(T, D).bfloat16(), rn(T, D).bfloat16(), nz(U, r), nz(U, D), nz(U, D)
    tau, isd, dden = torch.full((T,), 0.3, device=dev), torch.ones(T, device=dev), rn(T) * 0.01
    runs = []
    for _ in range(4):
        gr = [torch.zeros(U, d, device=dev) for d in (r, D, D)]
        dh, dx = torch.empty(T, r, device=dev), rn(T, D) * 0
        for _ in range(2):
            dtau = torch.zeros(T, device=dev)
            cb.ext().srw_route_bwd(x, h, tau, isd, dy, dden, dtau, emb, read, write, *gr, None, dh, True, dx,
                                   cb._gate_list(GateSpec(kind=1)), cb.status_word(dev))
        runs.append((dh, dx))
    cb.check_status()
    assert float(runs[0][1].abs().max()) > 0
    for dh, dx in runs[1:]:
        assert torch.equal(dh, runs[0][0]) and torch.equal(dx, runs[0][1])


@pytest.mark.parametrize("T,n,cols", [(1, 8, [(0, 8)]), (64, 128, [(0, 128)]), (65, 136, [(3, 130), (0, 136)]),
                                      (8192, 384, [(0, 384)]), (20011, 1160, [(0, 768), (768, 3), (768, 1)])])
def test_packed_gradient_and_its_column_sums_repeat(cb, T, n, cols):
    """One row block to many, ragged columns and rows: the bf16 operand exact, fp32 sums of T terms against
    fp64 (1e-5 of the terms' norm) and the same bits in every run."""
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(T)
    srcs = [torch.randn(T, w, device=dev, generator=g) for _, w in cols]
    total = torch.zeros(T, n, device=dev)
    for (c, w), s in zip(cols, srcs):
        total[:, c:c + w] += s
    first = None
    for _ in range(4):
        dst, db = cb.ext().linear_pack(srcs, [c for c, _ in cols], T, n, True, 0, 0.0, 0)
        first = db if first is None else first
        assert torch.equal(dst, total.bfloat16()) and torch.equal(db, first)
    assert float((db.double() - total.double().sum(0)).norm()) < 1e-5 * float(total.double().norm()) + 1e-6


def test_packed_gradient_of_more_rows_than_a_grid_has_blocks_of_64(cb):
    T, dev = 65535 * 64 + 77, torch.device("cuda")
    src = torch.randn(T, 8, device=dev)
    dst, db = cb.ext().linear_pack([src], [0], T, 8, True, 0, 0.0, 0)
    assert torch.equal(dst, src.bfloat16())
    assert float((db.double() - src.double().sum(0)).norm()) < 1e-5 * float(src.double().norm())


@pytest.mark.parametrize("T,D", [(1, 8), (9, 128), (8195, 136)])
def test_scale_gradient_of_a_route_repeats_bit_by_bit(cb, T, D):
    """Added to what is there; fp32 sums of T * D products against fp64: 1e-5 of their norm, sqrt(T)-fold for
    the sum over rows; the same bits in every run."""
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(T)
    dy, y, den = (torch.randn(*s, device=dev, generator=g) for s in ((T, D), (T, D), (T,)))
    scale, outs = torch.full((), 1.7, device=dev), []
    for _ in range(5):
        d_scale = torch.full((), 0.5, device=dev)
        cb.ext().route_bwd_rows(dy, y, den, 1.0, scale, None, torch.empty(T, device=dev), d_scale)
        outs.append(d_scale)
    dots = (dy.double() * y.double()).sum(-1) / 1.7
    assert abs(float(outs[0]) - 0.5 - float(dots.sum())) < 1e-5 * float(dots.norm()) * T ** 0.5 + 1e-5
    assert all(torch.equal(o, outs[0]) for o in outs)


@pytest.mark.parametrize("U,r", [(1, 8), (77, 512), (2600, 128), (100000, 256)])
def test_load_balance_gradient_repeats_bit_by_bit(cb, U, r):
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(U)
    emb = torch.randn(U, r, device=dev, generator=g).bfloat16()
    m_u = torch.randn(U, device=dev, generator=g)
    stat, one = torch.tensor([0.1, 1.2], device=dev), torch.ones((), device=dev)
    runs = [cb.ext().load_balance_bwd(emb, m_u, stat, one, 0.01, float(U)) for _ in range(4)]
    dmn, d_hsum = runs[0]
    want = dmn.double() @ emb.double()
    assert float((d_hsum.double() - want).norm()) < 1e-5 * float(dmn.norm()) * float(emb.double().norm()) / r ** 0.5
    assert all(torch.equal(a, dmn) and torch.equal(b, d_hsum) for a, b in runs[1:])


@pytest.mark.parametrize("T", [1, 40, 150])
def test_inference_call_takes_a_scale_on_the_host(cb, T):
    """The three regimes of row counts; a 0-dim tensor in host memory is a number like any other."""
    from dawn_srw_b200.ops.gates import GateSpec
    dev = torch.device("cuda")
    torch.manual_seed(T)
    U, r, D, be, spec = 600, 64, 128, cb.CudaBackend(), GateSpec(kind=1)
    pool = be.prepare_pool(*(torch.nn.functional.normalize(torch.randn(U, d, device=dev), dim=-1) for d in (r, D, D)),
                           spec)
    x, h, off = torch.randn(T, D, device=dev), torch.randn(T, 2, r, device=dev), torch.randn(T, 2, device=dev) * 0.1
    outs = [torch.stack(be.srw_infer(x, h, off, pool, spec, out_scale=s))
            for s in (0.75, torch.tensor(0.75), torch.tensor(0.75, device=dev), torch.tensor([0.75]))]
    cb.check_status()
    for o in outs[1:]:
        assert _rel(o, outs[0]) < 1e-5


@pytest.mark.parametrize("grad", [False, True])
def test_read_scalars_are_kept_only_for_a_backward_pass(cb, monkeypatch, grad):
    """With gradients enabled but nothing that requires one (a frozen model), no buffer is taken."""
    from dawn_srw_b200.ops.gates import GateSpec
    dev, kept = torch.device("cuda"), []
    U, r, D, T, be, spec = 2600, 64, 128, 300, cb.CudaBackend(), GateSpec(kind=1)
    alloc = cb._alloc_saved_xr
    monkeypatch.setattr(cb, "_alloc_saved_xr", lambda *a: kept.append(alloc(*a)) or kept[-1])
    pool = be.prepare_pool(*(torch.randn(U, d, device=dev) for d in (r, D, D)), spec)
    h = torch.randn(T, 1, r, device=dev, requires_grad=grad)
    be.srw(torch.randn(T, D, device=dev), h, torch.zeros(T, 1, device=dev), pool, spec, want_diag=False)
    assert len(kept) == 1 and (kept[0] is not None) == grad


def test_pool_call_without_tokens(cb):
    """Empty outputs, no gradient, and a load-balance term that is the mean over nothing."""
    from dawn_srw_b200.ops.gates import GateSpec
    dev = torch.device("cuda")
    U, r, D, be, spec = 600, 64, 128, cb.CudaBackend(), GateSpec(kind=1)
    ps = [torch.randn(U, d, device=dev, requires_grad=True) for d in (r, D, D)]
    x, h, off = (torch.empty(*s, device=dev, requires_grad=True) for s in ((0, D), (0, 2, r), (0, 2)))
    scale = torch.tensor(1.5, device=dev, requires_grad=True)
    res = be.srw(x, h, off, be.prepare_pool(*ps, spec), spec, want_diag=False, out_scale=scale)
    assert res.route(0).shape == (0, D) and bool(res.lb.isnan())
    (res.route(0).sum() + res.route(1).sum()).backward()
    cb.check_status()
    assert float(scale.grad) == 0.0 and all(float(p.grad.abs().max()) == 0.0 for p in ps)


def test_input_gradient_of_a_call_on_both_sides_of_its_summation_rule(cb):
    """dx of a two-route call just below and above the token count from which the routes' gradients are
    rounded to bf16 before they are added: rows of the same token agree to that rounding (2^-8 of the
    largest route, 8e-3 of the norm), and with fp64 of the formula to 2e-2 (bf16 operands)."""
    from dawn_srw_b200.ops.gates import GateSpec
    dev = torch.device("cuda")
    torch.manual_seed(5)
    D, r, U, be, spec = 256, 64, 600, cb.CudaBackend(), GateSpec(kind=1)
    T = next(t for t in range(256, 148 * 256, 256) if not cb.ext().gemm_few_tiles(t + 1, D))
    assert cb.ext().gemm_few_tiles(T, D) and not cb.ext().gemm_few_tiles(T + 1, D)
    ps = [torch.nn.functional.normalize(torch.randn(U, d, device=dev), dim=-1).requires_grad_(True) for d in (r, D, D)]
    x0, h, off = torch.randn(T + 1, D, device=dev), torch.randn(T + 1, 2, r, device=dev), torch.zeros(T + 1, 2, device=dev)
    dy, grads = torch.randn(2, T + 1, D, device=dev), []
    for t in (T, T + 1):
        x = x0[:t].clone().requires_grad_(True)
        res = be.srw(x, h[:t], off[:t], be.prepare_pool(*ps, spec), spec, want_diag=False, out_scale=1.0)
        sum((res.route(i) * dy[i, :t]).sum() for i in range(2)).backward()
        grads.append(x.grad)
    cb.check_status()
    assert float(grads[0].abs().max()) > 0 and _rel(grads[1][:T], grads[0]) < 8e-3


def test_layer_norm_gradients_of_more_rows_than_a_grid_has_blocks_of_64(cb):
    """fp32 sums of four million terms, added up by atomics of 64 and more rows: 1e-4 of the terms' norm."""
    T, D, dev = 65535 * 64 + 77, 4, torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(1)
    x, dy = torch.randn(T, D, device=dev, generator=g), torch.randn(T, D, device=dev, generator=g).bfloat16()
    w, b = torch.ones(D, device=dev, requires_grad=True), torch.zeros(D, device=dev, requires_grad=True)
    cb.CudaBackend().layer_norm(x, w, b).backward(dy)
    cb.check_status()
    xn = torch.nn.functional.layer_norm(x.double(), (D,), eps=1e-6)
    for got, terms in ((w.grad, dy.double() * xn), (b.grad, dy.double())):
        assert float((got.double() - terms.sum(0)).norm()) < 1e-4 * float(terms.norm())


@pytest.mark.parametrize("T,U,D,r", [(32, 19200, 384, 64), (33, 19200, 384, 64), (33, 1580, 384, 64), (64, 1580, 384, 64),
                                     (48, 6400, 1280, 64), (49, 6400, 1280, 64), (64, 6400, 2048, 64)])
def test_routes_on_both_sides_of_the_swapped_form(cb, T, U, D, r):
    """Where the rule by rows, units and width changes the form; the same bounds as between the forms."""
    test_route_of_a_few_rows_on_the_tensor_engine(cb, 1, T, U, D, r)


@pytest.mark.parametrize("M", [5, 16, 17, 24, 25, 32, 33, 48, 49, 64, 65])
def test_gemms_on_both_sides_of_the_swapped_form(cb, M):
    """One tile, one wave and more of them, short and long K, with and without a bias; fp32 sums, 1e-5."""
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(M)
    for N, K in ((8, 384), (128, 2048), (384, 384), (1280, 1280), (2048, 2048), (19200, 128), (384, 8192)):
        x, w = (torch.randn(n, K, device=dev, generator=g).bfloat16() for n in (M, N))
        for bias in (None, torch.randn(N, device=dev, generator=g)):
            ref = x.double() @ w.double().t() + (0.0 if bias is None else bias)
            assert _rel(cb.gemm(x, False, w, False, out_dtype=torch.float32, bias=bias), ref) < 1e-5
    cb.check_status()


@pytest.mark.parametrize("B,H,dh,S", [(1, 6, 64, 512), (6, 16, 128, 512), (2, 3, 36, 200)])
def test_decode_attention_around_the_positions_of_one_block(cb, B, H, dh, S):
    """Up to 96 cached positions the first CTA of a cluster works alone; fp32 sums in another order."""
    from dawn_srw_b200.ops import reference as R
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(dh)
    rn = lambda *s: torch.randn(*s, device=dev, generator=g)
    ck, cv, be = rn(B, H, S, dh), rn(B, H, S, dh), cb.CudaBackend()
    for pos in (2, 95, 96, 97, 128):
        q, k, v = rn(B, H * dh), rn(B, H * dh), rn(B, H * dh)
        out = be.decode_attention(q, k, v, ck, cv, torch.tensor([pos], device=dev), H)
        ref = R.cached_attention(q.view(B, H, 1, dh), ck, cv, pos + 1).reshape(B, H * dh)
        assert torch.equal(ck[:, :, pos].reshape(B, -1), k) and _rel(out, ref) < 1e-5


@pytest.mark.parametrize("T,D", [(16384, 384), (16385, 132), (70001, 8)])
def test_layer_norm_gradients_where_a_block_takes_more_rows(cb, T, D):
    """fp32 sums of T terms in another order: 1e-5 of the terms' norm."""
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(D)
    x, dy = torch.randn(T, D, device=dev, generator=g), torch.randn(T, D, device=dev, generator=g).bfloat16()
    w, b = torch.ones(D, device=dev, requires_grad=True), torch.zeros(D, device=dev, requires_grad=True)
    cb.CudaBackend().layer_norm(x, w, b).backward(dy)
    cb.check_status()
    xn = torch.nn.functional.layer_norm(x.double(), (D,), eps=1e-6)
    for got, terms in ((w.grad, dy.double() * xn), (b.grad, dy.double())):
        assert float((got.double() - terms.sum(0)).norm()) < 1e-5 * float(terms.norm())
