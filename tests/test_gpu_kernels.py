"""Parity of every sm_100a kernel, called through the C ABI, with an fp32 PyTorch statement
of the same operation on the same seeded inputs.  Tolerance: bf16 outputs within 2e-2 of
the reference magnitude; fp32 accumulations within 1e-3."""
import math

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def L():
    from bamboo_b200 import lib
    lib.load()
    return lib


def close(got, want, tol=2e-2):
    err = (got.float() - want.float()).abs().max().item()
    scale = want.float().abs().max().item()
    assert err <= tol * scale + 1e-3, (err, scale)


def gelu(x):
    return F.gelu(x, approximate="tanh")


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
@pytest.mark.parametrize("tile_n,cta_pair", [(128, -1), (256, -1), (0, 1)])
def test_gemm_operand_layouts(L, a_mn, b_mn, tile_n, cta_pair):
    torch.manual_seed(0)
    M, N, K = 384, 512, 320
    A = (torch.randn(M, K, device="cuda") * 0.5).bfloat16()
    B = (torch.randn(N, K, device="cuda") * 0.5).bfloat16()
    a = A.t().contiguous() if a_mn else A
    b = B.t().contiguous() if b_mn else B
    out = torch.zeros(M, N, device="cuda", dtype=torch.bfloat16)
    L.gemm(a, b, out, a_mn=a_mn, b_mn=b_mn, M=M, N=N, K=K, tile_n=tile_n, cta_pair=cta_pair)
    close(out, A.float() @ B.float().t())


@pytest.mark.parametrize("cta_pair", [-1, 1])
@pytest.mark.parametrize("shape", [(128, 128, 64), (200, 136, 72), (130, 264, 200), (8, 8, 8), (1024, 1024, 1000),
                                   (100, 260, 136), (520, 100, 72)])
def test_gemm_ragged_shapes(L, shape, cta_pair):
    """Edges: rows and columns that end inside a tile, inside a 16-byte store, or (pairs) before
    the second CTA's rows begin."""
    torch.manual_seed(1)
    M, N, K = shape
    A = torch.randn(M, K, device="cuda").bfloat16()
    B = torch.randn(N, K, device="cuda").bfloat16()
    bias = torch.randn(N + 8, device="cuda").bfloat16()[:N]
    ldd = (N + 7) // 8 * 8 + 8                                       # guard columns after N
    out = torch.full((M, ldd), 7.0, device="cuda", dtype=torch.bfloat16)
    L.gemm(A, B, out[:, :N], epilogue=L.EPI_BIAS, bias=bias, cta_pair=cta_pair)
    close(out[:, :N], A.float() @ B.float().t() + bias.float())
    assert torch.all(out[:, N:] == 7)                               # nothing written past column N
    aux = torch.randn(M, ldd, device="cuda").bfloat16()[:, :N]
    L.gemm(A, B, out[:, :N], epilogue=L.EPI_BIAS_RESIDUAL, bias=bias, aux=aux, cta_pair=cta_pair)
    close(out[:, :N], A.float() @ B.float().t() + bias.float() + aux.float())
    out.fill_(7)
    L.gemm(A, B, out[:, :N], epilogue=L.EPI_BIAS_RESIDUAL, bias=bias, aux=aux, cta_pair=cta_pair, epi_warps=4)
    close(out[:, :N], A.float() @ B.float().t() + bias.float() + aux.float())
    assert torch.all(out[:, N:] == 7)
    acc = torch.full((M, ldd), 7.0, device="cuda")
    L.gemm(A, B, acc[:, :N], epilogue=L.EPI_ACCUM_F32, cta_pair=cta_pair)
    close(acc[:, :N], A.float() @ B.float().t() + 7, 1e-3)
    assert torch.all(acc[:, N:] == 7)


@pytest.mark.parametrize("epi_warps", [2, 4])
@pytest.mark.parametrize("cta_pair", [-1, 1])
def test_gemm_epilogues(L, cta_pair, epi_warps):
    """Every fused epilogue, with 8 and with 16 epilogue warps (the latter bf16 outputs only)."""
    torch.manual_seed(2)
    M, N, K = 384, 768, 320
    A = (torch.randn(M, K, device="cuda") * 0.5).bfloat16()
    B = (torch.randn(N, K, device="cuda") * 0.5).bfloat16()
    bias = torch.randn(N, device="cuda").bfloat16()
    aux = torch.randn(M, N, device="cuda").bfloat16()
    ref = A.float() @ B.float().t()
    out = torch.zeros(M, N, device="cuda", dtype=torch.bfloat16)
    out2 = torch.zeros_like(out)
    L.gemm(A, B, out, epilogue=L.EPI_BIAS_GELU, bias=bias, out2=out2, cta_pair=cta_pair, epi_warps=epi_warps)
    close(out2, ref + bias.float())
    close(out, gelu((ref + bias.float()).bfloat16().float()))
    L.gemm(A, B, out, epilogue=L.EPI_BIAS_RESIDUAL, bias=bias, aux=aux, cta_pair=cta_pair, epi_warps=epi_warps)
    close(out, ref + bias.float() + aux.float())
    x = aux.float().requires_grad_(True)
    gelu(x).sum().backward()
    L.gemm(A, B, out, epilogue=L.EPI_MUL_DGELU, aux=aux, cta_pair=cta_pair, epi_warps=epi_warps)
    close(out, ref * x.grad)
    acc = torch.randn(M, N, device="cuda")
    want = acc + ref
    L.gemm(A, B, acc, epilogue=L.EPI_ACCUM_F32, cta_pair=cta_pair)
    close(acc, want, 1e-3)
    L.gemm(A, B, acc, epilogue=L.EPI_STORE_F32, cta_pair=cta_pair)
    close(acc, ref, 1e-3)


def test_gemm_is_linear_and_deterministic_at_full_size(L):
    """GPT-2-medium MLP shape: two runs are bit-identical and (A1+A2)B = A1 B + A2 B in fp32 output."""
    torch.manual_seed(3)
    M, N, K = 8192, 4096, 1024
    A1 = torch.randint(-4, 5, (M, K), device="cuda").bfloat16()
    A2 = torch.randint(-4, 5, (M, K), device="cuda").bfloat16()
    B = torch.randint(-4, 5, (N, K), device="cuda").bfloat16()
    o1, o2, o12, again = (torch.empty(M, N, device="cuda") for _ in range(4))
    L.gemm(A1, B, o1, epilogue=L.EPI_STORE_F32)
    L.gemm(A2, B, o2, epilogue=L.EPI_STORE_F32)
    L.gemm((A1 + A2), B, o12, epilogue=L.EPI_STORE_F32)
    L.gemm(A1, B, again, epilogue=L.EPI_STORE_F32)
    assert torch.equal(o1, again)
    assert torch.equal(o12, o1 + o2)          # small integers: exact in bf16 x bf16 -> fp32
    assert torch.equal(o1[:256], (A1[:256].float() @ B.float().t()))


def test_gemm_cta_pairs_at_full_size(L):
    """Input-gradient shape of the MLP (long reduction, B stored [K, N]): the heuristic picks CTA
    pairs; small integers make the result exact, and single CTAs must give the same bits."""
    torch.manual_seed(13)
    M, N, K = 8192, 1024, 4096
    A = torch.randint(-3, 4, (M, K), device="cuda").bfloat16()
    B = torch.randint(-3, 4, (K, N), device="cuda").bfloat16()      # stored [K, N]
    pair = torch.empty(M, N, device="cuda")
    single = torch.empty(M, N, device="cuda")
    L.gemm(A, B, pair, b_mn=True, epilogue=L.EPI_STORE_F32, M=M, N=N, K=K)
    L.gemm(A, B, single, b_mn=True, epilogue=L.EPI_STORE_F32, M=M, N=N, K=K, cta_pair=-1)
    assert torch.equal(pair, single)
    assert torch.equal(pair[:512], A[:512].float() @ B.float())


@pytest.mark.parametrize("cta_pair", [-1, 1])
@pytest.mark.parametrize("split", [0, 1, 3, 8])
def test_gemm_split_k_accumulation(L, split, cta_pair):
    """Weight-gradient shape (few output tiles, long reduction): partial sums of the K splits
    meet in the fp32 add-reduction."""
    torch.manual_seed(11)
    M, N, K = 1024, 1024, 8192
    A = torch.randint(-3, 4, (K, M), device="cuda").bfloat16()      # stored [K, M]
    B = torch.randint(-3, 4, (K, N), device="cuda").bfloat16()      # stored [K, N]
    acc = torch.ones(M, N, device="cuda")
    L.gemm(A, B, acc, a_mn=True, b_mn=True, epilogue=L.EPI_ACCUM_F32, M=M, N=N, K=K, split_k=split, cta_pair=cta_pair)
    want = A.float().t() @ B.float() + 1
    assert torch.equal(acc, want)                                    # small integers: exact


# (output channels, columns, rows of the reduction): one to many output tiles, reductions of one k-block, of a few (left
# whole), and of so many that a single tile is split over the whole machine; ragged last splits and pairs
@pytest.mark.parametrize("M,N,K", [(64, 64, 40), (8, 72, 130), (128, 128, 800), (64, 392, 4097), (64, 64, 100352), (256, 2304, 1000),
                                   (1024, 256, 64), (256, 512, 25088), (512, 4608, 2100)])
def test_gemm_planned_weight_gradients(L, M, N, K):
    """The add-reduction epilogue with tile, pairing and split left to the library, on top of existing gradients,
    against fp64.  Products of bf16 values are exact in fp32; what differs is the fp32 rounding of the sums: with
    random signs about sqrt(K) additions of 2^-24 each, 2e-5 at the longest reduction."""
    g = torch.Generator(device="cuda").manual_seed(3)
    a = torch.randn(K, M, device="cuda", generator=g).bfloat16()
    b = torch.randn(K, N, device="cuda", generator=g).bfloat16()
    start = torch.randn(M, N, device="cuda", generator=g)
    d = start.clone()
    for _ in range(2):
        L.gemm(a, b, d, a_mn=True, b_mn=True, epilogue=L.EPI_ACCUM_F32, M=M, N=N, K=K)
    want = start.double() + 2 * (a.double().t() @ b.double())
    err = ((d.double() - want).norm() / want.norm()).item()
    print(f"weight gradient {M}x{N}x{K}: relative error {err:.2e}")
    assert err <= 2e-5
    assert L.read_status() == 0


def test_gemm_rejects_bad_arguments(L):
    A = torch.zeros(16, 12, device="cuda", dtype=torch.bfloat16)   # leading dimension not a multiple of 8
    B = torch.zeros(16, 12, device="cuda", dtype=torch.bfloat16)
    out = torch.zeros(16, 16, device="cuda", dtype=torch.bfloat16)
    with pytest.raises(L.BambooNativeError):
        L.gemm(A, B, out)
    with pytest.raises(L.BambooNativeError):
        L.gemm(out, out, out, epilogue=L.EPI_BIAS)                 # bias missing
    with pytest.raises(L.BambooNativeError):
        L.gemm(out, out, torch.zeros(16, 16, device="cuda"), epilogue=L.EPI_STORE_F32, epi_warps=4)   # fp32 output


@pytest.mark.parametrize("rows,h", [(512, 256), (8192, 1024), (300, 768), (1000, 4096)])
def test_layernorm(L, rows, h):
    torch.manual_seed(4)
    x = torch.randn(rows, h, device="cuda").bfloat16()
    g = (1 + 0.1 * torch.randn(h, device="cuda")).bfloat16()
    b = (0.1 * torch.randn(h, device="cuda")).bfloat16()
    y = torch.empty_like(x)
    mean, rstd = torch.empty(rows, device="cuda"), torch.empty(rows, device="cuda")
    L.layernorm_fwd(x, g, b, y, mean, rstd, 1e-5)
    xf, gf, bf = x.float().requires_grad_(True), g.float().requires_grad_(True), b.float().requires_grad_(True)
    yr = F.layer_norm(xf, (h,), gf, bf, 1e-5)
    close(y, yr)
    dy, dres = torch.randn(rows, h, device="cuda").bfloat16(), torch.randn(rows, h, device="cuda").bfloat16()
    yr.backward(dy.float())
    dx = torch.empty_like(x)
    dg, db = torch.ones(h, device="cuda"), torch.ones(h, device="cuda")      # accumulate on top of 1
    L.layernorm_bwd(dy, x, g, mean, rstd, dres, dx, dg, db)
    close(dx, xf.grad + dres.float())
    close(dg - 1, gf.grad)
    close(db - 1, bf.grad)


@pytest.mark.parametrize("rows,h", [(8192, 1024), (777, 256), (300, 768), (1000, 2048), (515, 4096), (64, 8192), (100, 1000)])
def test_layernorm_backward_with_residual_sums(L, rows, h):
    """One pass gives dx, dgamma, dbeta and the column sums of the residual gradient; every
    column-owner instantiation (hidden sizes up to 1024, 2048, 4096, 8192) and the fallback."""
    torch.manual_seed(6)
    x = torch.randn(rows, h, device="cuda").bfloat16()
    g = (1 + 0.1 * torch.randn(h, device="cuda")).bfloat16()
    b = torch.zeros(h, device="cuda").bfloat16()
    y = torch.empty_like(x)
    mean, rstd = torch.empty(rows, device="cuda"), torch.empty(rows, device="cuda")
    L.layernorm_fwd(x, g, b, y, mean, rstd, 1e-5)
    dy, dres = torch.randn(rows, h, device="cuda").bfloat16(), torch.randn(rows, h, device="cuda").bfloat16()
    dx0, dx1 = torch.empty_like(x), torch.empty_like(x)
    dg0, db0 = torch.zeros(h, device="cuda"), torch.zeros(h, device="cuda")
    dg1, db1, ds1 = torch.zeros(h, device="cuda"), torch.zeros(h, device="cuda"), torch.ones(h, device="cuda")
    L.layernorm_bwd(dy, x, g, mean, rstd, dres, dx0, dg0, db0)
    L.layernorm_bwd_res(dy, x, g, mean, rstd, dres, dx1, dg1, db1, ds1)
    close(dx1, dx0, 1e-2)
    close(dg1, dg0, 1e-4)
    close(db1, db0, 1e-4)
    close(ds1 - 1, dres.float().sum(0), 1e-3)
    xf, gf = x.float().requires_grad_(True), g.float().requires_grad_(True)
    F.layer_norm(xf, (h,), gf, b.float(), 1e-5).backward(dy.float())
    close(dx1, xf.grad + dres.float())
    close(dg1, gf.grad)
    # in place over the residual gradient
    alias = dres.clone()
    ds2 = torch.zeros(h, device="cuda")
    L.layernorm_bwd_res(dy, x, g, mean, rstd, alias, alias, dg1, db1, ds2)
    close(alias, dx1, 1e-2)
    close(ds2, dres.float().sum(0), 1e-3)
    assert L.read_status() == 0


@pytest.mark.parametrize("rows,n", [(8192, 4096), (8192, 1024), (100, 264), (513, 1024), (1, 8), (4096, 50304), (33, 3072)])
def test_colsum(L, rows, n):
    torch.manual_seed(5)
    dy = torch.randn(rows, n, device="cuda").bfloat16()
    out = torch.ones(n, device="cuda")
    L.colsum_accum(dy, out)
    close(out - 1, dy.float().sum(0), 1e-3)
    # the ticket counters return to zero: repeated calls (also back to back on two streams, each
    # with its own scratch) give the same bits
    again = torch.ones(n, device="cuda")
    L.colsum_accum(dy, again)
    assert torch.equal(out, again)
    side = torch.cuda.Stream()
    a, b = torch.zeros(n, device="cuda"), torch.zeros(n, device="cuda")
    torch.cuda.synchronize()
    for _ in range(3):
        L.colsum_accum(dy, a)
        with torch.cuda.stream(side):
            L.colsum_accum(dy, b, tag="test-side", stream=side.cuda_stream)
    torch.cuda.synchronize()
    assert torch.equal(a, b)
    close(a, 3 * dy.float().sum(0), 1e-3)


def test_gelu_backward(L):
    torch.manual_seed(4)
    pre = torch.randn(1000, 1024, device="cuda").bfloat16()
    dy = torch.randn_like(pre)
    dx = torch.empty_like(pre)
    L.gelu_bwd(dy, pre, dx)
    x = pre.float().requires_grad_(True)
    gelu(x).backward(dy.float())
    close(dx, x.grad)


def test_embedding(L):
    torch.manual_seed(6)
    V, h, B, S = 1024, 256, 4, 128
    tok = torch.randint(0, V, (B, S), device="cuda")
    tok[0, :8] = 7                                                   # collisions in the scatter
    wte, wpe = torch.randn(V, h, device="cuda").bfloat16(), torch.randn(S, h, device="cuda").bfloat16()
    out = torch.empty(B * S, h, device="cuda", dtype=torch.bfloat16)
    L.embedding_fwd(tok, wte, wpe, out, S)
    close(out, wte[tok.view(-1)].float() + wpe.float().repeat(B, 1))
    dout = torch.randn(B * S, h, device="cuda").bfloat16()
    dwte, dwpe = torch.zeros(V, h, device="cuda"), torch.zeros(S, h, device="cuda")
    L.embedding_bwd(tok, dout, dwte, dwpe, S)
    close(dwte, torch.zeros(V, h, device="cuda").index_add_(0, tok.view(-1), dout.float()), 1e-3)
    close(dwpe, dout.float().view(B, S, h).sum(0), 1e-3)


@pytest.mark.parametrize("rows,V,Vp", [(512, 1024, 1024), (1024, 50257, 50304), (100, 30522, 30528), (4, 8, 8)])
def test_cross_entropy(L, rows, V, Vp):
    torch.manual_seed(7)
    logits = torch.zeros(rows, Vp, device="cuda", dtype=torch.bfloat16)
    logits[:, :V] = (3 * torch.randn(rows, V, device="cuda")).bfloat16()
    tgt = torch.randint(0, V, (rows,), device="cuda")
    tgt[::7] = -100                                                  # ignored positions
    lse, rl, lo = torch.empty(rows, device="cuda"), torch.empty(rows, device="cuda"), torch.empty(2, device="cuda")
    L.cross_entropy_fwd(logits, tgt, lse, rl, lo, V)
    lf = logits[:, :V].float().requires_grad_(True)
    ref = F.cross_entropy(lf, tgt, ignore_index=-100)
    assert lo[0].item() == pytest.approx(ref.item(), rel=1e-4)
    assert lo[1].item() == (tgt != -100).sum().item()
    (ref * 0.25).backward()
    L.cross_entropy_bwd(logits, tgt, lse, lo, logits, V, grad_scale=0.25)       # in place
    close(logits[:, :V], lf.grad)
    assert logits[:, V:].abs().max().item() == 0 if Vp > V else True


def test_adam_matches_torch(L):
    torch.manual_seed(8)
    n = 1 << 20
    p, m, v = torch.randn(n, device="cuda"), torch.zeros(n, device="cuda"), torch.zeros(n, device="cuda")
    g, lp = torch.empty(n, device="cuda"), torch.empty(n, device="cuda", dtype=torch.bfloat16)
    pr = p.clone().requires_grad_(True)
    opt = torch.optim.Adam([pr], lr=1e-3)
    for step in (1, 2, 3):
        gg = torch.randn(n, device="cuda")
        g.copy_(gg)
        pr.grad = gg.clone()
        opt.step()
        L.adam_step(p, g, m, v, lp, lr=1e-3, step=step)
    close(p, pr.detach(), 1e-5)
    close(lp, pr.detach(), 1e-2)
    assert g.abs().max().item() == 0
    close(m, opt.state[pr]["exp_avg"], 1e-5)
    close(v, opt.state[pr]["exp_avg_sq"], 1e-5)


def _attn_ref(qkv, B, H, S, D, causal):
    q, k, v = qkv.float().view(B, S, 3, H, D).permute(2, 0, 3, 1, 4)
    return F.scaled_dot_product_attention(q, k, v, is_causal=causal).permute(0, 2, 1, 3).reshape(B * S, H * D)


@pytest.mark.parametrize("B,H,S,D,causal", [(2, 4, 128, 64, True), (2, 3, 256, 64, False), (1, 2, 1024, 64, True),
                                            (1, 2, 200, 64, True), (1, 2, 72, 64, False), (1, 2, 256, 128, True),
                                            (2, 2, 320, 128, False),
                                            # an odd number of 64-query sub-blocks (the fused backward pairs them up and
                                            # pads with a masked one that reads the next batch's rows), several key tiles
                                            (2, 2, 192, 64, True), (2, 2, 192, 64, False), (2, 1, 448, 64, True),
                                            (1, 1, 2048, 64, True), (3, 2, 640, 64, False),
                                            # head dimension 128: tcgen05 forward (two 64-column atoms per row), warp-level backward
                                            (1, 2, 1024, 128, True), (1, 2, 200, 128, True), (2, 1, 448, 128, False),
                                            (1, 1, 72, 128, False),
                                            (1, 16, 2048, 128, True)])     # enough CTAs to keep every SM and the TMA unit busy
def test_attention(L, B, H, S, D, causal):
    torch.manual_seed(9)
    qkv = torch.randn(B * S, 3 * H * D, device="cuda").bfloat16()
    out = torch.empty(B * S, H * D, device="cuda", dtype=torch.bfloat16)
    lse = torch.empty(B, H, S, device="cuda")
    L.attention_fwd(qkv, out, lse, B, H, S, D, causal)
    qf = qkv.float().requires_grad_(True)
    ref = _attn_ref(qf, B, H, S, D, causal)
    close(out, ref)
    do = torch.randn_like(out)
    ref.backward(do.float())
    dqkv = torch.empty_like(qkv)
    L.attention_bwd(qkv, out, do, lse, dqkv, B, H, S, D, causal)
    close(dqkv, qf.grad)


def test_attention_backward_with_fixed_summation_order(L):
    """BB_ATTENTION_BWD=split selects the two-role backward kernels (dK/dV and dQ by different CTAs, no
    reductions into an accumulator): same gradients, and bit-identical from run to run.  The switch is read
    once per process, so the check runs in a child process."""
    import os
    import subprocess
    import sys
    code = """
import sys, torch
sys.path.insert(0, %r)
import torch.nn.functional as F
from bamboo_b200 import lib as L
L.load()
B, H, S, D = 2, 2, 448, 64
torch.manual_seed(3)
qkv = torch.randn(B * S, 3 * H * D, device="cuda").bfloat16()
out = torch.empty(B * S, H * D, device="cuda", dtype=torch.bfloat16)
lse = torch.empty(B, H, S, device="cuda")
L.attention_fwd(qkv, out, lse, B, H, S, D, True)
qf = qkv.float().requires_grad_(True)
q, k, v = qf.view(B, S, 3, H, D).permute(2, 0, 3, 1, 4)
ref = F.scaled_dot_product_attention(q, k, v, is_causal=True).permute(0, 2, 1, 3).reshape(B * S, H * D)
do = torch.randn_like(out)
ref.backward(do.float())
a, b = torch.empty_like(qkv), torch.empty_like(qkv)
L.attention_bwd(qkv, out, do, lse, a, B, H, S, D, True)
L.attention_bwd(qkv, out, do, lse, b, B, H, S, D, True)
torch.cuda.synchronize()
err = (a.float() - qf.grad).abs().max().item()
assert err <= 2e-2 * qf.grad.abs().max().item() + 1e-3, err
assert torch.equal(a, b)
assert L.read_status() == 0
print("split backward ok")
""" % os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, BB_ATTENTION_BWD="split")
    r = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "split backward ok" in r.stdout, r.stdout + r.stderr


def test_attention_rows_sum_to_one_at_full_size(L):
    """GPT-2-medium attention shape: with V = 1 every output element must be 1."""
    B, H, S, D = 8, 16, 1024, 64
    torch.manual_seed(10)
    qkv = torch.randn(B * S, 3 * H * D, device="cuda").bfloat16()
    qkv[:, 2 * H * D:] = 1
    out = torch.empty(B * S, H * D, device="cuda", dtype=torch.bfloat16)
    lse = torch.empty(B, H, S, device="cuda")
    L.attention_fwd(qkv, out, lse, B, H, S, D, True)
    assert (out.float() - 1).abs().max().item() < 1e-2
    assert torch.isfinite(lse).all()


def test_attention_backward_checksums_at_full_size(L):
    """GPT-2-medium attention shape, properties that hold at any size: every probability row sums
    to one, so the V-gradient summed over keys equals dO summed over queries; and the score
    gradient of a row sums to zero, so with all keys equal the Q-gradient vanishes."""
    B, H, S, D = 8, 16, 1024, 64
    torch.manual_seed(12)
    qkv = (torch.randn(B * S, 3 * H * D, device="cuda") * 0.5).bfloat16()
    qkv[:, H * D:2 * H * D] = qkv[0, H * D:2 * H * D]               # the same key vector at every position
    out = torch.empty(B * S, H * D, device="cuda", dtype=torch.bfloat16)
    lse = torch.empty(B, H, S, device="cuda")
    L.attention_fwd(qkv, out, lse, B, H, S, D, True)
    do = torch.randn_like(out)
    dqkv = torch.empty_like(qkv)
    L.attention_bwd(qkv, out, do, lse, dqkv, B, H, S, D, True)
    dq, dv = dqkv[:, :H * D].float(), dqkv[:, 2 * H * D:].float()
    want = do.float().view(B, S, H * D).sum(1)
    got = dv.view(B, S, H * D).sum(1)
    assert (got - want).abs().max().item() <= 2e-2 * want.abs().max().item() + 0.5   # bf16 rounding of 1024 addends
    assert dq.abs().max().item() <= 2e-2 * do.float().abs().max().item()
    assert L.read_status() == 0


def test_ping_counter_may_run_ahead_of_the_receiver(L):
    """A liveness ping carries no payload: its flag is a counter.  A receiver that waits for ping
    1 after the sender already signalled ping 3 has its answer (lazy redundancy on more than two
    stages does exactly that); a payload slot whose flag moved on is an error, and a ping that
    never comes ends the bounded wait with the peer-timeout status.  All on this GPU's own memory."""
    import ctypes
    lib = L.load()
    flag = torch.zeros(1, dtype=torch.int64, device="cuda")
    stream = L._stream()
    fp = ctypes.c_void_p(flag.data_ptr())
    assert lib.bb_p2p_signal(fp, ctypes.c_ulonglong(3), stream) == 0
    assert lib.bb_p2p_wait_copy(None, None, ctypes.c_longlong(0), fp, ctypes.c_ulonglong(1),
                                ctypes.c_ulonglong(200_000_000), None, stream) == 0
    torch.cuda.synchronize()
    assert L.read_status() == 0
    src = torch.ones(64, device="cuda"); dst = torch.zeros(64, device="cuda")
    assert lib.bb_p2p_wait_copy(ctypes.c_void_p(src.data_ptr()), ctypes.c_void_p(dst.data_ptr()), ctypes.c_longlong(256), fp,
                                ctypes.c_ulonglong(1), ctypes.c_ulonglong(200_000_000), None, stream) == 0
    torch.cuda.synchronize()
    assert L.read_status() == -1 and float(dst.sum()) == 0          # overwritten slot: reported, nothing copied
    assert lib.bb_p2p_wait_copy(None, None, ctypes.c_longlong(0), fp, ctypes.c_ulonglong(9),
                                ctypes.c_ulonglong(50_000_000), None, stream) == 0
    torch.cuda.synchronize()
    assert L.read_status() == L.STATUS_PEER_TIMEOUT                   # the wait ran out, the context lives on
    assert L.read_status() == 0


def test_status_word_is_clean(L):
    torch.cuda.synchronize()
    assert L.read_status() == 0


# Head dimension 128 backward on the tensor cores, at the edges of its 128-row tiles and 64-row sub-blocks: one row, one
# short of / one past a sub-block and a tile, several batches (a partial tile reads the next batch's rows, masked).
# Tolerance: bf16 P and dS carry 2^-9 relative error each, sums are fp32 - the 2e-2 of `close` is an order above.
@pytest.mark.parametrize("B,H,S,causal", [(2, 1, 1, True), (2, 2, 63, False), (2, 2, 65, True), (3, 1, 127, True),
                                          (2, 3, 129, False), (2, 1, 257, True), (1, 2, 385, False)])
def test_attention_backward_head_dim_128_tile_edges(L, B, H, S, causal):
    D = 128
    torch.manual_seed(21)
    qkv = torch.randn(B * S, 3 * H * D, device="cuda").bfloat16()
    out = torch.empty(B * S, H * D, device="cuda", dtype=torch.bfloat16)
    lse = torch.empty(B, H, S, device="cuda")
    L.attention_fwd(qkv, out, lse, B, H, S, D, causal)
    qf = qkv.float().requires_grad_(True)
    ref = _attn_ref(qf, B, H, S, D, causal)
    do = torch.randn_like(out)
    ref.backward(do.float())
    dqkv = torch.full_like(qkv, float("nan"))
    L.attention_bwd(qkv, out, do, lse, dqkv, B, H, S, D, causal)
    again = torch.full_like(qkv, float("nan"))
    L.attention_bwd(qkv, out, do, lse, again, B, H, S, D, causal)
    close(dqkv, qf.grad)
    assert torch.equal(dqkv, again)                     # every sum in a fixed order
    assert L.read_status() == 0


# Head dimension 64 at the edges of its 128-row tiles and 64-key sub-blocks, and with scores that grow along the keys
# (grow > 0: the running maximum outgrows the exponent reference again and again, so the accumulator row in tensor
# memory is rescaled between the products).  Tolerance as above; the log-sum-exp is
# fp32 throughout: 1e-3 absolute covers the bf16 rounding of nothing but the inputs' products (exact in fp32) and ex2 / log2.
@pytest.mark.parametrize("B,H,S,causal,grow", [(2, 1, 1, True, 0.0), (2, 1, 63, False, 0.0), (2, 2, 65, True, 0.0),
                                               (3, 1, 127, True, 0.0), (2, 3, 129, False, 0.0), (2, 1, 257, True, 0.0),
                                               (1, 2, 385, False, 0.0), (5, 7, 191, True, 0.0), (1, 2, 320, True, 0.05),
                                               (1, 2, 449, False, 0.05), (2, 16, 777, True, 0.02)])
def test_attention_head_dim_64_tile_edges(L, B, H, S, causal, grow):
    D = 64
    torch.manual_seed(22)
    qkv = torch.randn(B * S, 3 * H * D, device="cuda")
    if grow:
        k = qkv[:, H * D:2 * H * D].view(B, S, H * D)
        k *= 1.0 + grow * torch.arange(S, device="cuda").view(1, S, 1)
    qkv = qkv.bfloat16()
    out = torch.full((B * S, H * D), float("nan"), device="cuda", dtype=torch.bfloat16)
    lse = torch.full((B, H, S), float("nan"), device="cuda")
    L.attention_fwd(qkv, out, lse, B, H, S, D, causal)
    qf = qkv.float().requires_grad_(True)
    ref = _attn_ref(qf, B, H, S, D, causal)
    close(out, ref)
    q, k = (qkv[:, i * H * D:(i + 1) * H * D].double().view(B, S, H, D).transpose(1, 2) for i in range(2))
    scores = q @ k.transpose(-1, -2) / D ** 0.5
    if causal:
        scores.masked_fill_(torch.ones(S, S, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
    want = torch.logsumexp(scores, -1)
    assert ((lse.double() - want).abs() / (1.0 + want.abs())).max().item() <= 1e-3
    do = torch.randn_like(out)
    ref.backward(do.float())
    dqkv = torch.full_like(qkv, float("nan"))
    L.attention_bwd(qkv, out, do, lse, dqkv, B, H, S, D, causal)
    close(dqkv, qf.grad)
    assert L.read_status() == 0


@pytest.mark.parametrize("B,H,S,causal,want_out,want_lse",
                         [(2, 3, 257, False, "9a5419f9f8e4b22c", "28ec0ae142d23f85"), (1, 2, 1000, True, "17536437b67bc51e", "0507974505271b4a"),
                          (3, 1, 64, True, "30ae10657d9dc1ad", "2a728876a08dc590")])
def test_attention_head_dim_64_keeps_its_summation_order(L, B, H, S, causal, want_out, want_lse):
    """Output and log-sum-exp in every bit: digests of what the two-tile kernel (one CTA per 256 query rows), which had this
    head dimension before, gives for the same inputs.  A row's sum takes columns i and i + 32 of a sub-block together,
    i ascending; any other order changes last bits of the log-sum-exp and, after a few layers, every activation."""
    import hashlib
    D = 64
    i = torch.arange(B * S * 3 * H * D)
    qkv = ((i * 2654435761 % 65521).float() / 65521 * 4 - 2).view(B * S, 3 * H * D).bfloat16().cuda()
    out = torch.empty(B * S, H * D, device="cuda", dtype=torch.bfloat16)
    lse = torch.empty(B, H, S, device="cuda")
    L.attention_fwd(qkv, out, lse, B, H, S, D, causal)
    digest = [hashlib.sha256(t.cpu().view(torch.uint8).numpy().tobytes()).hexdigest()[:16] for t in (out, lse)]
    assert digest == [want_out, want_lse]


# lengths that end inside a 64-row sub-block, inside a 128-row tile, and one past a tile (the next tile of the machine then
# lies almost wholly past the end); 384: no overhang, for the heads' own accumulator rows
@pytest.mark.parametrize("S", [1, 50, 100, 129, 300, 384])
@pytest.mark.parametrize("D,causal", [(64, True), (64, False), (128, True), (128, False)])
def test_attention_non_finite_values_stay_in_their_sequence(L, D, causal, S):
    """A tile that overhangs the end of a sequence must not let in its neighbour's rows, nor add to its neighbour's: zero
    (a masked probability) times Inf is NaN.  One head of the middle sequence is Inf / NaN; every other (sequence, head)
    has to come out as without it - the same bits, but for dQ at head dimension 64, whose additions have no fixed
    order (bf16 result: 2^-8 of the largest value)."""
    B, H = 3, 3
    torch.manual_seed(31)
    clean = torch.randn(B, S, 3, H, D, device="cuda").bfloat16()
    dclean = torch.randn(B, S, H, D, device="cuda").bfloat16()
    bad, dbad = clean.clone(), dclean.clone()
    bad[1, :, 0, 1], bad[1, :, 1, 1], bad[1, :, 2, 1] = float("inf"), float("nan"), float("inf")
    dbad[1, :, 1] = float("inf")

    def passes(qkv, do):
        qkv, do = qkv.reshape(B * S, 3 * H * D), do.reshape(B * S, H * D)
        out = torch.empty(B * S, H * D, device="cuda", dtype=torch.bfloat16)
        lse = torch.empty(B, H, S, device="cuda")
        dqkv = torch.empty_like(qkv)
        L.attention_fwd(qkv, out, lse, B, H, S, D, causal)
        L.attention_bwd(qkv, out, do, lse, dqkv, B, H, S, D, causal)
        return out.view(B, S, H, D), lse, dqkv.view(B, S, 3, H, D)

    (o0, l0, g0), (o1, l1, g1) = passes(clean, dclean), passes(bad, dbad)
    assert not torch.isfinite(o1[1, :, 1].float()).all()
    for b in range(B):
        for h in range(H):
            if (b, h) == (1, 1):
                continue
            assert torch.equal(o0[b, :, h], o1[b, :, h]) and torch.equal(l0[b, h], l1[b, h]), (b, h)
            assert torch.equal(g0[b, :, 1:, h], g1[b, :, 1:, h]), (b, h)
            if D == 128:
                assert torch.equal(g0[b, :, 0, h], g1[b, :, 0, h]), (b, h)
            else:
                assert ((g0[b, :, 0, h].float() - g1[b, :, 0, h].float()).abs().max() <= 2 ** -8 * g0[b, :, 0, h].float().abs().max()).item(), (b, h)
    assert L.read_status() == 0


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
@pytest.mark.parametrize("tile_n,cta_pair", [(128, -1), (256, -1), (0, 1)])
@pytest.mark.parametrize("shape", [(8, 8, 8), (128, 128, 64), (136, 264, 200), (304, 520, 1000), (520, 1032, 2048)])
def test_gemm_reduction_split_inside_a_cluster(L, a_mn, b_mn, tile_n, cta_pair, shape):
    """Every number of splits (more than panels or k-blocks among them) with every bf16 epilogue, operand layout and a leading
    dimension of its own.  Operands of -1, 0 and 1: sums are whole numbers below 2^24, the same in any order, so the stored value is
    the bf16 rounding of the fp32 result bit for bit."""
    torch.manual_seed(21)
    M, N, K = shape
    A = torch.randint(-1, 2, (M, K), device="cuda").bfloat16()
    B = torch.randint(-1, 2, (N, K), device="cuda").bfloat16()
    a, b = A.t().contiguous() if a_mn else A, B.t().contiguous() if b_mn else B
    bias = torch.randint(-4, 5, (N,), device="cuda").bfloat16()
    aux = torch.randint(-4, 5, (M, N + 8), device="cuda").bfloat16()[:, :N]
    ref = A.float() @ B.float().t()
    wide = torch.empty(M, N + 8, device="cuda", dtype=torch.bfloat16)
    out, pre = wide[:, :N], torch.empty(M, N + 8, device="cuda", dtype=torch.bfloat16)[:, :N]
    for split in (1, 2, 3, 4, 5, 6, 7, 8, 40):
        kw = dict(a_mn=a_mn, b_mn=b_mn, M=M, N=N, K=K, tile_n=tile_n, cta_pair=cta_pair, split_k=split)
        wide.fill_(7)
        L.gemm(a, b, out, **kw)
        assert torch.equal(out, ref.bfloat16()) and torch.all(wide[:, N:] == 7)
        L.gemm(a, b, out, epilogue=L.EPI_BIAS_RESIDUAL, bias=bias, aux=aux, **kw)
        assert torch.equal(out, (ref + bias.float() + aux.float()).bfloat16())
        L.gemm(a, b, out, epilogue=L.EPI_BIAS_GELU, bias=bias, out2=pre, **kw)
        assert torch.equal(pre, (ref + bias.float()).bfloat16())
        close(out, gelu(pre.float()))
    assert L.read_status() == 0


@pytest.mark.parametrize("shape", [(520, 2048, 4096), (64, 2048, 2048), (1000, 512, 2048), (136, 1032, 4104)])
def test_gemm_planned_split_is_as_exact_as_the_whole_reduction(L, shape):
    """Shapes whose plan splits the reduction: the distance from 64 bits is that of one chain of additions, or less (both end in
    one bf16 rounding, which dominates: the larger of the two may exceed the other by the fp32 part, 2^-24 sqrt(K) relative)."""
    torch.manual_seed(22)
    M, N, K = shape
    A, B = torch.randn(M, K, device="cuda").bfloat16(), torch.randn(N, K, device="cuda").bfloat16()
    ref = A.double() @ B.double().t()
    out, whole = (torch.empty(M, N, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    L.gemm(A, B, out)
    L.gemm(A, B, whole, tile_n=128, cta_pair=-1)
    err = [float((o.double() - ref).norm() / ref.norm()) for o in (out, whole)]
    assert err[0] <= err[1] + 2 ** -24 * K ** 0.5


@pytest.mark.parametrize("tile_n,cta_pair", [(128, -1), (256, -1), (0, 1)])
@pytest.mark.parametrize("accum", [False, True])
def test_gemm_of_several_waves_in_a_graph(L, tile_n, cta_pair, accum):
    """More work units than CTAs, captured once and replayed on new operands, with calls outside the graph in between: every
    replay computes every tile.  Whole numbers: sums are exact in any order."""
    torch.manual_seed(23)
    M, N, K = (4168, 2312, 136) if not accum else (2312, 2056, 1032)
    A, B = torch.zeros(M, K, device="cuda", dtype=torch.bfloat16), torch.zeros(N, K, device="cuda", dtype=torch.bfloat16)
    out = torch.zeros(M, N, device="cuda", dtype=torch.float32 if accum else torch.bfloat16)
    kw = dict(tile_n=tile_n, cta_pair=cta_pair, epilogue=L.EPI_ACCUM_F32 if accum else L.EPI_STORE, split_k=2 if accum else 0)
    L.gemm(A, B, out, **kw)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        L.gemm(A, B, out, **kw)
    for _ in range(3):
        for t in (A, B):
            t.copy_(torch.randint(-1, 2, t.shape, device="cuda"))
        ref = A.float() @ B.float().t()
        ref = ref if accum else ref.bfloat16()
        for run in (graph.replay, lambda: L.gemm(A, B, out, **kw)):
            out.zero_()
            run()
            assert torch.equal(out, ref)
    assert L.read_status() == 0


@pytest.mark.parametrize("limit", [dict(max_ctas=16), dict(max_ctas=-1), dict(epi_warps=2), dict(max_ctas=6, cta_pair=1), dict(max_ctas=100000)])
def test_gemm_budget_goes_before_a_split_of_the_reduction(L, limit):
    """A descriptor that names a split of a bf16 product together with a cap on its CTAs keeps the cap: the same launch, and the same
    bits, as without the split.  (A cap above the number of SMs is none.)"""
    from cuda.bindings import driver
    from test_gpu_overlap import captured, kernel_nodes
    torch.manual_seed(24)
    M, N, K = 520, 1032, 2048
    A, B = torch.randn(M, K, device="cuda").bfloat16(), torch.randn(N, K, device="cuda").bfloat16()
    out = [torch.empty(M, N, device="cuda", dtype=torch.bfloat16) for _ in range(2)]
    shapes = []
    for split in (0, 4):
        graph, handle, rt = captured(lambda: L.gemm(A, B, out[split > 0], split_k=split, **limit))
        node, = kernel_nodes(handle, rt)
        cluster = rt.cudaGraphKernelNodeGetAttribute(node, rt.cudaLaunchAttributeID.cudaLaunchAttributeClusterDimension)[1].clusterDim.x
        shapes.append((driver.cuGraphKernelNodeGetParams(driver.CUgraphNode(int(node)))[1].gridDimX, cluster))
    if limit.get("max_ctas", 0) > 1000:
        assert shapes[1][1] >= 4
    else:
        assert shapes[0] == shapes[1] and (limit.get("max_ctas", 0) <= 0 or shapes[1][0] <= limit["max_ctas"])
        assert torch.equal(*out)


# outputs just below and at 2^22 elements, with panels inside the matrix and across its edges; 4 bytes a column in a longer row
@pytest.mark.parametrize("M,N", [(2040, 2048), (2048, 2048), (2056, 2060), (130, 32268)])
@pytest.mark.parametrize("tile_n,cta_pair", [(128, -1), (256, -1), (0, 1)])
def test_gemm_add_reduction_into_small_and_large_outputs(L, M, N, tile_n, cta_pair):
    """Whole numbers: sums are exact in any order, and what lies beside the matrix is not touched."""
    torch.manual_seed(25)
    K = 200
    A, B = (torch.randint(-1, 2, (K, n + (-n) % 8), device="cuda").bfloat16() for n in (M, N))
    wide = torch.full((M + 1, N + 4), 3.0, device="cuda")
    for split in (1, 2):
        L.gemm(A, B, wide[:M, :N], a_mn=True, b_mn=True, epilogue=L.EPI_ACCUM_F32, M=M, N=N, K=K, tile_n=tile_n, cta_pair=cta_pair, split_k=split)
    want = torch.full_like(wide, 3.0)
    want[:M, :N] += 2 * (A[:, :M].float().t() @ B[:, :N].float())
    assert torch.equal(wide, want)
    assert L.read_status() == 0


@pytest.mark.parametrize("tile_n,cta_pair", [(128, -1), (256, -1), (0, 1)])
@pytest.mark.parametrize("shape", [(8, 8, 72), (136, 264, 200), (520, 1032, 2048)])
def test_gemm_split_inside_a_cluster_with_bias_and_gelu_derivative(L, tile_n, cta_pair, shape):
    """The two bf16 epilogues that the test of all splits leaves out.  Sums of whole numbers are the same in any order, and what is done to
    them is the same code: the bits of the whole reduction."""
    torch.manual_seed(26)
    M, N, K = shape
    A, B = torch.randint(-1, 2, (M, K), device="cuda").bfloat16(), torch.randint(-1, 2, (N, K), device="cuda").bfloat16()
    bias, aux = torch.randint(-4, 5, (N,), device="cuda").bfloat16(), (2 * torch.randn(M, N + 8, device="cuda")).bfloat16()[:, :N]
    want = (A.float() @ B.float().t() + bias.float()).bfloat16()
    out, whole = (torch.empty(M, N, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    kw = dict(tile_n=tile_n, cta_pair=cta_pair)
    L.gemm(A, B, whole, epilogue=L.EPI_MUL_DGELU, aux=aux, **kw)
    for split in (1, 2, 3, 4, 5, 6, 7, 8, 40):
        L.gemm(A, B, out.fill_(7), epilogue=L.EPI_BIAS, bias=bias, split_k=split, **kw)
        assert torch.equal(out, want)
        L.gemm(A, B, out.fill_(7), epilogue=L.EPI_MUL_DGELU, aux=aux, split_k=split, **kw)
        assert torch.equal(out, whole)
    assert L.read_status() == 0


def split_launch(call):
    """Whether the call's one product runs with its reduction split over clusters: that kernel has 608 threads, the other 352."""
    from cuda.bindings import driver
    from test_gpu_overlap import captured, kernel_nodes
    graph, handle, rt = captured(call)
    node, = kernel_nodes(handle, rt)
    return driver.cuGraphKernelNodeGetParams(driver.CUgraphNode(int(node)))[1].blockDimX == 608


@pytest.mark.parametrize("shape", [(520, 2048, 4096), (64, 2048, 2048), (1000, 512, 2048), (136, 1032, 4104)])
@pytest.mark.parametrize("budget", [-1, 64])
def test_gemm_own_and_redundant_routes_agree(L, shape, budget):
    """The stage's own product splits its reduction, the same product on the CTA budget of redundant work keeps it whole: sums that are
    exact in any order give the same bits; others are as far from 64 bits either way (one bf16 rounding, and the fp32
    part of 2^-24 sqrt(K))."""
    torch.manual_seed(27)
    M, N, K = shape
    out = [torch.empty(M, N, device="cuda", dtype=torch.bfloat16) for _ in range(2)]
    for exact in (True, False):
        A, B = ((torch.randint(-1, 2, (n, K), device="cuda") if exact else torch.randn(n, K, device="cuda")).bfloat16() for n in (M, N))
        calls = [lambda: L.gemm(A, B, out[0]), lambda: L.gemm(A, B, out[1], max_ctas=budget)]
        assert [split_launch(c) for c in calls] == [True, False]
        for c in calls:
            c()
        ref = A.double() @ B.double().t()
        if exact:
            assert torch.equal(out[0], ref.bfloat16()) and torch.equal(*out)
        else:
            err = [float((o.double() - ref).norm() / ref.norm()) for o in out]
            assert abs(err[0] - err[1]) <= 2 ** -24 * K ** 0.5
