"""Numerics of every sm_100a kernel against the fp32 PyTorch restatement of the same op."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

from vllm_cpp_b200 import ops  # noqa: E402
from vllm_cpp_b200.ops import reference as ref  # noqa: E402
from vllm_cpp_b200.ops._lib import KernelError  # noqa: E402

DEV = "cuda"


def _rand(*shape, scale=1.0, dtype=torch.bfloat16):
    return (torch.randn(*shape, device=DEV, dtype=torch.float32) * scale).to(dtype)


from _numerics import rel_err as _rel_err  # noqa: E402


def test_library_loaded_and_status_clean():
    assert ops.num_sms() >= 100
    assert ops.read_status() == 0


@pytest.mark.parametrize("M,N,K", [(128, 256, 64), (512, 1024, 512), (300, 520, 328),
                                   (1024, 4096, 4096), (4096, 6144, 4096), (257, 128, 8192)])
@pytest.mark.parametrize("path", [3, 4])
def test_gemm_tiled(M, N, K, path):
    torch.manual_seed(0)
    a, w = _rand(M, K), _rand(N, K, scale=0.05)
    out = ops.gemm(a, w, force_path=path)
    exp = ref.gemm(a, w)
    assert _rel_err(out, exp) < 6e-3
    assert ops.read_status() == 0


@pytest.mark.parametrize("M,N,K", [(1280, 4096, 4096), (1280, 4096, 14336), (384, 4096, 4096),
                                   (1000, 6144, 4096), (130, 512, 8192), (520, 4104, 1024),
                                   (128, 256, 64)])
@pytest.mark.parametrize("path", [0, 5, 6])
def test_gemm_stream_k(M, N, K, path):
    """Stream-K: tiles are cut along K across CTAs and fixed up through fp32 partials. Run twice:
    the second launch only works if the first one cleared every flag it consumed."""
    torch.manual_seed(2)
    a, w = _rand(M, K), _rand(N, K, scale=0.05)
    r = _rand(M, N)
    exp = ref.gemm(a, w)
    for _ in range(2):
        out = ops.gemm(a, w, force_path=path)
        assert _rel_err(out, exp) < 6e-3
    out = ops.gemm(a, w, residual=r, force_path=path, out_dtype=torch.float32)
    assert _rel_err(out, exp + r.float()) < 6e-3
    assert ops.read_status() == 0


@pytest.mark.parametrize("M,N,K", [(1, 4096, 4096), (8, 6144, 4096), (16, 128, 64), (33, 4096, 14336),
                                   (64, 28672, 4096), (200, 1024, 1024), (256, 4096, 4096),
                                   (5, 128256, 1024), (1, 28672, 4096), (17, 32768, 512), (64, 16384, 192)])
def test_gemm_small_m_swap_splitk(M, N, K):
    torch.manual_seed(1)
    a, w = _rand(M, K), _rand(N, K, scale=0.05)
    out = ops.gemm(a, w)
    exp = ref.gemm(a, w)
    assert _rel_err(out, exp) < 6e-3
    assert ops.read_status() == 0


@pytest.mark.parametrize("M,N,K", [(32, 4096, 4096), (64, 28672, 4096), (200, 1024, 1024), (1280, 4096, 4096)])
def test_gemm_const_weight_early_fetch_in_a_chain(M, N, K):
    """``const_w`` lets the GEMM fetch weight tiles before the previous kernel has finished; the
    activations still have to wait for it. A chain norm -> GEMM -> norm -> GEMM, launched back to
    back, must give the same bits as the same chain without the flag."""
    torch.manual_seed(11)
    x0 = _rand(M, K)
    g = _rand(K)
    w1 = _rand(N, K, scale=0.05)
    w2 = _rand(K, N, scale=0.02)

    def chain(flag):
        x = x0
        for _ in range(3):
            h = ops.rmsnorm(x, g, 1e-6)
            y = ops.gemm(h, w1, const_w=flag)
            x = ops.gemm(y, w2, const_w=flag)
        return x

    a, b = chain(False), chain(True)
    assert torch.equal(a, b)
    h = ops.rmsnorm(x0, g, 1e-6)
    assert _rel_err(ops.gemm(h, w1, const_w=True), ref.gemm(h, w1)) < 6e-3
    assert ops.read_status() == 0


def test_gemm_epilogues():
    torch.manual_seed(2)
    for M in (7, 700):
        a, w = _rand(M, 512), _rand(768, 512, scale=0.05)
        bias, res = _rand(768), _rand(M, 768)
        out = ops.gemm(a, w, bias=bias, residual=res)
        assert _rel_err(out, ref.gemm(a, w, bias, res)) < 6e-3
        o32 = ops.gemm(a, w, out_dtype=torch.float32)
        assert o32.dtype == torch.float32
        assert _rel_err(o32, ref.gemm(a, w, out_dtype=torch.float32)) < 2e-3
    # strided activations (a column slice of a wider buffer)
    big = _rand(300, 1024)
    a = big[:, 256:768]
    w = _rand(384, 512, scale=0.05)
    assert _rel_err(ops.gemm(a, w), ref.gemm(a, w)) < 6e-3
    assert ops.read_status() == 0


@pytest.mark.parametrize("M", [1, 16, 17, 48, 127, 128])
@pytest.mark.parametrize("N,K", [(8, 64), (136, 72), (128, 512), (1032, 1000), (6144, 1024)])
def test_gemm_over_a_cluster(M, N, K):
    """Up to 128 rows, K in 1 to 8 parts over a cluster: edges of row tiles and of k-blocks, every number of parts, what
    follows the product. A value is off by its rounding to bf16 at most (8 significant bits: 2^-8), in 32 bits by the sums' order."""
    torch.manual_seed(M * 7 + N + K)
    a, w = _rand(M, K + 8)[:, :K], _rand(N, K, scale=0.05)
    bias, res = _rand(N), _rand(M, N + 8)[:, :N]
    exact = a.double() @ w.double().t()
    for parts in (0, 1, 2, 3, 5, 8):
        path = 32 + parts if parts else 0
        o32 = ops.gemm(a, w, out_dtype=torch.float32, force_path=path)
        assert _rel_err(o32.double(), exact) < 5e-5
        assert _rel_err(ops.gemm(a, w, force_path=path).double(), exact) < 2.0 ** -8
        both = ops.gemm(a, w, bias=bias, residual=res, force_path=path)
        assert _rel_err(both.double(), exact + bias.double() + res.double()) < 2.0 ** -8
    act = ops.gemm(a, w, act=4)
    assert _rel_err(act.double(), exact.clamp_min(0).square()) < 2.0 ** -8
    assert ops.read_status() == 0


@pytest.mark.parametrize("M", [1, 33, 128])
@pytest.mark.parametrize("I,K", [(128, 64), (384, 200), (3072, 1024)])
def test_gemm_gated_over_a_cluster(M, I, K):
    torch.manual_seed(M + I)
    a, g, u = _rand(M, K), _rand(I, K, scale=0.05), _rand(I, K, scale=0.05)
    for kind in (0, 1, 2):
        out = ops.gemm_gated(a, ops.interleave_gate_up(g, u), kind)
        merged = ops.gemm(a, torch.cat([g, u], 0), force_path=1)           # rounded before the activation, as here
        exp = ref.act_and_mul(merged, kind)
        assert _rel_err(out, exp) < 2.0 ** -6      # gate, up and their product are rounded once each (3 x 2^-8)
    assert ops.read_status() == 0


@pytest.mark.parametrize("M,I,apart", [(32, 19200, 0), (33, 19200, 1), (96, 9600, 0), (97, 9600, 1), (128, 16000, 0), (129, 19200, 0)])
def test_gemm_gated_in_one_and_in_two_kernels(M, I, apart):
    """Both sides of the lines, against 64 bits: gate, up and their product are rounded once each (3 x 2^-8, and the sums)."""
    from vllm_cpp_b200.ops import _lib
    torch.manual_seed(M)
    K = 264
    assert bool(_lib.lib().b200_gemm_gated_apart(M, 2 * I)) == bool(apart)
    a, g, u = _rand(M, K), _rand(I, K, scale=0.05), _rand(I, K, scale=0.05)
    w = ops.interleave_gate_up(g, u)
    gd, ud = a.double() @ g.double().t(), a.double() @ u.double().t()
    exp = gd * torch.sigmoid(gd) * ud
    forms = [ops.gemm_gated(a, w)] + ([ops.gemm_gated(a, w, force_path=32)] if M <= 128 else [])
    room = torch.full((M, I + 8), 7.0, dtype=torch.bfloat16, device=DEV)
    forms.append(ops.gemm_gated(a, w, out=room[:, :I]))                # rows of its own pitch: one kernel
    for out in forms:
        assert _rel_err(out.double(), exp) < 2.0 ** -6
    assert bool((room[:, I:] == 7.0).all()) and ops.read_status() == 0


@pytest.mark.parametrize("M", [1, 2])
@pytest.mark.parametrize("N,K", [(8, 8), (264, 72), (1032, 1000), (6144, 1024), (4096, 14336), (40000, 512)])
def test_gemm_of_one_or_two_rows(M, N, K):
    """Warp-wide products: ragged chunks of K, one to eight warps a pair of rows, several turns of a block. Off by the
    rounding to bf16 at most (2^-8)."""
    torch.manual_seed(M + N)
    a, w = _rand(M, K + 8)[:, :K], _rand(N, K, scale=0.05)
    bias, res = _rand(N), _rand(M, N + 8)[:, :N]
    exact = a.double() @ w.double().t()
    assert _rel_err(ops.gemm(a, w, out_dtype=torch.float32).double(), exact) < 5e-6 * K ** 0.5
    assert _rel_err(ops.gemm(a, w, const_w=True).double(), exact) < 2.0 ** -8
    assert _rel_err(ops.gemm(a, w, bias=bias, residual=res).double(), exact + bias.double() + res.double()) < 2.0 ** -8
    assert _rel_err(ops.gemm(a, w, act=4).double(), exact.clamp_min(0).square()) < 2.0 ** -8
    assert ops.read_status() == 0


@pytest.mark.parametrize("M,N,K", [(3, 8192, 256), (3, 8064, 264), (1, 7104, 136), (1, 7112, 136), (2, 14208, 520), (2, 14216, 520),
                                   (1, 21312, 1000), (1, 21320, 1000), (16, 38016, 512), (17, 38016, 512), (17, 38016, 520)])
def test_gemm_at_the_lines_between_its_forms(M, N, K):
    """Turns of a block of one- and two-row products, four k-blocks in one part, wide matrices with a short K. Off by the
    rounding to bf16 at most (2^-8)."""
    torch.manual_seed(N + K)
    a, w = _rand(M, K), _rand(N, K, scale=0.05)
    assert _rel_err(ops.gemm(a, w).double(), a.double() @ w.double().t()) < 2.0 ** -8
    assert ops.read_status() == 0


@pytest.mark.parametrize("M,N,K", [(1, 1032, 264), (40, 1032, 2048), (17, 16400, 264), (40, 16400, 264), (200, 1032, 2048), (200, 16400, 264),
                                   (300, 1032, 264), (600, 16400, 264)])
def test_gemm_with_bias_and_residual_at_any_address(M, N, K):
    """Every form reads them in pieces of its own size: addresses that are multiples of 16, 8 and 2 bytes. A tiling that was
    asked for and cannot read them refuses."""
    torch.manual_seed(M + N)
    a, w = _rand(M, K), _rand(N, K, scale=0.05)
    bias, res = _rand(N + 8), _rand(M * N + 8)
    exact = a.double() @ w.double().t()
    for off in (0, 4, 1):
        b, r = bias[off: off + N], res[off: off + M * N].view(M, N)
        assert _rel_err(ops.gemm(a, w, bias=b).double(), exact + b.double()) < 2.0 ** -8
        assert _rel_err(ops.gemm(a, w, bias=bias[:N], residual=r).double(), exact + bias[:N].double() + r.double()) < 2.0 ** -8
        if off:
            with pytest.raises(KernelError):
                ops.gemm(a, w, bias=b, force_path=7)
    assert ops.read_status() == 0


def test_gemm_deterministic():
    torch.manual_seed(3)
    a, w = _rand(48, 4096), _rand(4096, 4096, scale=0.05)
    o1 = ops.gemm(a, w).clone()
    o2 = ops.gemm(a, w)
    assert torch.equal(o1, o2)


@pytest.mark.parametrize("T,H", [(1, 1024), (37, 4096), (5, 5120), (3, 2048)])
def test_rmsnorm(T, H):
    torch.manual_seed(4)
    x, w, r = _rand(T, H), _rand(H), _rand(T, H)
    out = ops.rmsnorm(x, w, 1e-6)
    exp, _ = ref.rmsnorm(x, w, 1e-6)
    assert _rel_err(out, exp) < 5e-3
    r2 = r.clone()
    out = ops.rmsnorm(x, w, 1e-6, residual=r2, gemma=True)
    exp, newr = ref.rmsnorm(x, w, 1e-6, residual=r, gemma=True)
    assert torch.equal(r2, newr)
    assert _rel_err(out, exp) < 5e-3


def test_layernorm_and_eltwise():
    torch.manual_seed(5)
    x, w, b = _rand(9, 768), _rand(768), _rand(768)
    assert _rel_err(ops.layernorm(x, w, b, 1e-5), ref.layernorm(x, w, b, 1e-5)) < 5e-3
    a, c = _rand(16, 512), _rand(16, 512)
    assert _rel_err(ops.add(a, c), (a.float() + c.float())) < 5e-3
    assert torch.equal(ops.relu(a), torch.relu(a))
    assert _rel_err(ops.mul_scalar(a, 0.37), a.float() * 0.37) < 5e-3
    assert _rel_err(ops.softcap(a, 30.0), 30.0 * torch.tanh(a.float() / 30.0)) < 5e-3
    assert _rel_err(ops.sigmoid_mul(a, c), a.float() * torch.sigmoid(c.float())) < 5e-3
    assert torch.equal(ops.cast_bf16(ops.cast_f32(a)), a)


@pytest.mark.parametrize("kind", [0, 1, 2])
def test_act_and_mul(kind):
    torch.manual_seed(6)
    x = _rand(33, 2 * 1408)
    assert _rel_err(ops.act_and_mul(x, kind), ref.act_and_mul(x, kind)) < 5e-3


def _all_bf16():
    return torch.arange(-32768, 32768, device=DEV).to(torch.int16).view(torch.bfloat16)


@pytest.mark.parametrize("scale", [0.0, 1.0])
def test_silu_of_every_gate(scale):
    """act(gate) * up for all 65536 gates, up 1 and 31 random values: the result lies between the roundings of what the arithmetic may
    err by, so mostly it is the correctly rounded one. __expf: 2 + 1.173 |x| units of 2^-23, times its share in the result; the
    quotient and the product with up: 2^-22 and 2^-24, the bounds' own rounding to 32 bits as much. Beyond 32 bits' range: 2e-36."""
    torch.manual_seed(4)
    gate = _all_bf16()[None].expand(32, -1)
    up = torch.exp2(torch.randn(32, 65536, device=DEV) * scale * 3).to(torch.bfloat16)
    got = ops.act_and_mul(torch.cat([gate, up], 1).contiguous(), 0)
    g, u = gate.double(), up.double()
    e = torch.exp(-g.abs())
    exact = g * u * torch.where(g >= 0, 1.0, e) / (1 + e)
    part = torch.where(g >= 0, e, torch.ones_like(e)) / (1 + e)
    err = (2 + 1.173 * g.abs()) * 2.0 ** -23 * part + 2.0 ** -22 + 2 * 2.0 ** -24
    low, high = ((exact.abs() * (1 + s * err)).to(torch.bfloat16).double() for s in (-1, 1))
    at, size = torch.isfinite(g) & torch.isfinite(high), got.double().abs()
    fine = ((size >= low) & (size <= high)) | ((size - exact.abs()).abs() <= 2e-36 * u.clamp_min(1.0))
    assert bool(fine[at].all())
    assert torch.equal(torch.signbit(got[at]), torch.signbit(g[at]))                  # (zeros, and what underflows)
    right = exact.to(torch.bfloat16) == got
    assert (~right[at & (g.abs() < 20)]).double().mean().item() < 2.0 ** -10            # (the bounds are that much of a step of 2^-8)
    assert bool((got[gate == float("inf")] == float("inf")).all())
    assert bool(torch.isnan(got[torch.isnan(gate) | (gate == -float("inf"))]).all())


@pytest.mark.parametrize("M", [2, 40, 128, 256])
def test_silu_of_every_gate_in_a_products_epilogue(M):
    """The same bits where a product applies it: gates that a unit row picks out of the weights."""
    gate = _all_bf16().view(256, 256)
    gate = torch.where(torch.isfinite(gate), gate, torch.zeros_like(gate))
    up = torch.ones_like(gate)
    a = torch.eye(256, device=DEV, dtype=torch.bfloat16)[:M]
    got = ops.gemm_gated(a, ops.interleave_gate_up(gate, up))
    exp = ops.act_and_mul(torch.cat([gate.t()[:M], up[:M]], 1).contiguous(), 0)
    assert torch.equal(got, exp) and ops.read_status() == 0


def test_embedding_and_gather():
    torch.manual_seed(7)
    table = _rand(1000, 256)
    ids = torch.randint(0, 1000, (77,), device=DEV)
    assert torch.equal(ops.embedding(ids, table), table[ids])
    # vocab shard: rows outside are zero, no error flag
    out = ops.embedding(ids, table[500:], vocab_start=500, vocab_total=1000)
    exp = torch.where((ids >= 500)[:, None], table[ids], torch.zeros_like(table[ids]))
    assert torch.equal(out, exp)
    assert ops.read_status() == 0
    bad = ids.clone()
    bad[3] = 5000
    ops.embedding(bad, table)
    assert ops.read_status() == 3  # flagged, no fault
    assert ops.read_status() == 0
    idx = torch.randint(0, 77, (13,), device=DEV, dtype=torch.int32)
    x = _rand(77, 256)
    assert torch.equal(ops.gather_rows(x, idx), x[idx.long()])


@pytest.mark.parametrize("neox,rot,qk_norm", [(True, 128, False), (True, 128, True),
                                              (False, 64, False), (True, 64, True)])
def test_rope_kv(neox, rot, qk_norm):
    torch.manual_seed(8)
    T, Hq, Hkv, D, bs, nb = 45, 8, 2, 128, 16, 12
    qkv = _rand(T, (Hq + 2 * Hkv) * D)
    pos = torch.randint(0, 500, (T,), device=DEV)
    inv = ref.rope_inv_freq(rot, 1e6).to(DEV)
    table = ops.rope_table(inv, 512)
    assert torch.allclose(table, ref.rope_table(inv, 512), atol=2e-6)
    qn = _rand(D) if qk_norm else None
    kn = _rand(D) if qk_norm else None
    slots = torch.randperm(nb * bs, device=DEV)[:T].to(torch.int64)
    slots[5] = -1
    cache = torch.zeros(nb, 2, bs, Hkv, D, device=DEV, dtype=torch.bfloat16)
    eq, ek, ev = ref.rope_kv(qkv, pos, table, Hq, Hkv, D, rot, neox, qn, kn)
    work = qkv.clone()
    ops.rope_kv(work, pos, table, num_q_heads=Hq, num_kv_heads=Hkv, head_dim=D, rot_dim=rot,
                neox=neox, q_norm=qn, k_norm=kn, slot_mapping=slots, kv_cache=cache, block_size=bs)
    got_q = work[:, : Hq * D].reshape(T, Hq, D)
    assert _rel_err(got_q, eq) < 8e-3
    exp_cache = torch.zeros_like(cache)
    ref.write_kv_cache(exp_cache, ek, ev, slots, bs)
    assert _rel_err(cache[:, 0], exp_cache[:, 0]) < 8e-3
    assert torch.equal(cache[:, 1], exp_cache[:, 1])


def _make_paged(seq_lens, Hkv, D, bs, extra_blocks=3):
    nb_per = [(s + bs - 1) // bs for s in seq_lens]
    total = sum(nb_per) + extra_blocks
    cache = _rand(total, 2, bs, Hkv, D)
    perm = torch.randperm(total, device=DEV).to(torch.int32)
    maxb = max(nb_per)
    bt = torch.zeros(len(seq_lens), maxb, dtype=torch.int32, device=DEV)
    o = 0
    for r, n in enumerate(nb_per):
        bt[r, :n] = perm[o:o + n]
        o += n
    return cache, bt


@pytest.mark.parametrize("D,Hq,Hkv,bs", [(128, 8, 2, 16), (128, 4, 4, 32), (64, 4, 1, 16),
                                         (128, 4, 1, 128), (256, 6, 1, 16), (256, 2, 2, 64)])
def test_attn_prefill(D, Hq, Hkv, bs):
    torch.manual_seed(9)
    q_lens = [200, 17, 128, 333]
    ctx = [0, 40, 256, 77]  # cached prefix per request (chunked prefill / prefix hit)
    seq_lens = [a + b for a, b in zip(q_lens, ctx)]
    cache, bt = _make_paged(seq_lens, Hkv, D, bs)
    T = sum(q_lens)
    q = _rand(T, Hq * D)
    qs = torch.tensor([0] + list(torch.tensor(q_lens).cumsum(0)), dtype=torch.int32, device=DEV)
    sl = torch.tensor(seq_lens, dtype=torch.int32, device=DEV)
    treq, tq0 = ref.build_prefill_tiles(q_lens)
    treq = torch.tensor(treq, dtype=torch.int32, device=DEV)
    tq0 = torch.tensor(tq0, dtype=torch.int32, device=DEV)
    scale = D ** -0.5
    lse = torch.empty(T, Hq, dtype=torch.float32, device=DEV)
    out = ops.attn_prefill(q, cache, block_table=bt, seq_lens=sl, q_start=qs, tile_req=treq,
                           tile_q0=tq0, num_q_heads=Hq, num_kv_heads=Hkv, head_dim=D,
                           block_size=bs, scale=scale, lse=lse)
    exp, exp_lse = ref.paged_attention(q, cache, bt, sl, qs, Hq, Hkv, D, bs, scale, return_lse=True)
    assert ops.read_status() == 0
    assert _rel_err(out, exp) < 1.5e-2
    assert torch.allclose(lse, exp_lse, atol=2e-2, rtol=1e-3)


@pytest.mark.parametrize("Hq,Hkv,bs,window,causal,peak", [(4, 2, 8, 0, True, 1.0), (8, 1, 256, 0, True, 8.0), (12, 2, 32, 150, True, 1.0),
                                                          (8, 4, 64, -200, True, 1.0), (4, 2, 16, 0, False, 8.0),
                                                          (12, 2, 32, 1024, True, 1.0), (8, 4, 64, -1100, True, 1.0)])
def test_attn_prefill_head_pairs(Hq, Hkv, bs, window, causal, peak):
    """128-dim heads in even groups: edges of the 128-row and 128-key tiles, cached prefixes, windows and chunks, keys that
    raise a row's maximum late (``peak``: the later half of the keys is that much longer). P and the output are rounded to
    bf16 once each (2 x 2^-8). Enough tiles and, as the kernel is told, keys for two heads a CTA, except for the short
    windows."""
    torch.manual_seed(Hq + bs)
    D, q_lens, ctx = 128, [1, 127, 128, 129, 300, 4200], [400, 0, 128, 1, 513, 0]
    assert Hq * sum(-(-n // 128) for n in q_lens) > ops.num_sms()
    seq_lens = [a + b for a, b in zip(q_lens, ctx)]
    cache, bt = _make_paged(seq_lens, Hkv, D, bs)
    for r, n in enumerate(seq_lens):
        cache[bt[r, (n + bs - 1) // bs // 2: (n + bs - 1) // bs].long(), 0] *= peak
    T = sum(q_lens)
    q = _rand(T, Hq * D + 64)[:, :Hq * D]
    qs = torch.tensor([0] + list(torch.tensor(q_lens).cumsum(0)), dtype=torch.int32, device=DEV)
    sl = torch.tensor(seq_lens, dtype=torch.int32, device=DEV)
    treq, tq0 = ref.build_prefill_tiles(q_lens)
    lse = torch.empty(T, Hq, dtype=torch.float32, device=DEV)
    out = ops.attn_prefill(q, cache, block_table=bt, seq_lens=sl, q_start=qs, tile_req=torch.tensor(treq, dtype=torch.int32, device=DEV),
                           tile_q0=torch.tensor(tq0, dtype=torch.int32, device=DEV), num_q_heads=Hq, num_kv_heads=Hkv, head_dim=D,
                           block_size=bs, scale=D ** -0.5, window=window, causal=causal, lse=lse, tile_keys=10 ** 6)
    G = Hq // Hkv
    for r, (n, c) in enumerate(zip(q_lens, ctx)):
        rows = slice(int(qs[r]), int(qs[r]) + n)
        k, v = (cache[bt[r].long(), i].reshape(-1, Hkv, D)[: n + c].double().repeat_interleave(G, 1) for i in (0, 1))
        score = torch.einsum("qhd,khd->hqk", q[rows].reshape(n, Hq, D).double(), k) * D ** -0.5
        i, j = torch.arange(c, c + n, device=DEV)[:, None], torch.arange(n + c, device=DEV)[None]
        see = (j <= i) if causal else torch.ones_like(j <= i)
        if window > 0:
            see &= j > i - window
        elif window < 0:
            see &= j >= i // -window * -window
        score = score.masked_fill(~see, -float("inf"))
        exp = torch.einsum("hqk,khd->qhd", torch.softmax(score, -1), v)
        got = out[rows].view(n, Hq, D).double()
        assert ((got - exp).norm() / exp.norm()).item() < 2 * 2.0 ** -8
        assert (lse[rows].double().t() - torch.logsumexp(score, -1)).abs().max().item() < 1e-3
    assert ops.read_status() == 0


@pytest.mark.parametrize("n,L", [(1, 400), (20, 130), (6, 384), (6, 383)])
def test_attn_prefill_one_and_two_heads_a_cta(n, L):
    """Both sides of the rule, told the number of keys or left to guess it: the rounding of P and the output (2 x 2^-8)."""
    torch.manual_seed(L)
    D, Hq, Hkv, bs = 128, 16, 4, 32
    cache, bt = _make_paged([L] * n, Hkv, D, bs)
    q = _rand(n * L, Hq * D)
    treq, tq0 = ref.build_prefill_tiles([L] * n)
    I = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)       # noqa: E731
    kw = dict(block_table=bt, seq_lens=I([L] * n), q_start=I([i * L for i in range(n + 1)]), tile_req=I(treq), tile_q0=I(tq0),
              num_q_heads=Hq, num_kv_heads=Hkv, head_dim=D, block_size=bs, scale=D ** -0.5)
    keys = n * sum(min(a + 128, L) for a in range(0, L, 128))
    outs = [ops.attn_prefill(q, cache, tile_keys=r, **kw).double() for r in (keys, 0, 1, 10 ** 6)]
    k, v = (cache[bt.long(), i].reshape(n, -1, Hkv, D)[:, :L].double().repeat_interleave(Hq // Hkv, 2) for i in (0, 1))
    score = torch.einsum("nqhd,nkhd->nhqk", q.view(n, L, Hq, D).double(), k) * D ** -0.5
    score = score.masked_fill(torch.ones(L, L, dtype=torch.bool, device=DEV).triu(1), -float("inf"))
    exp = torch.einsum("nhqk,nkhd->nqhd", torch.softmax(score, -1), v).reshape(n * L, Hq * D)
    for got in outs:
        assert ((got - exp).norm() / exp.norm()).item() < 2 * 2.0 ** -8
    assert ops.read_status() == 0


@pytest.mark.parametrize("splits", [3, 12288, 12289])
def test_attn_decode_of_very_many_splits(splits):
    """The merge of split partials with its weights in shared memory and, beyond what that holds, without; most splits are
    empty. fp32 throughout, one rounding to bf16."""
    torch.manual_seed(splits)
    D, Hq, Hkv, bs = 64, 4, 2, 16
    cache, bt = _make_paged([300, 17], Hkv, D, bs)
    q = _rand(2, Hq * D)
    sl = torch.tensor([300, 17], dtype=torch.int32, device=DEV)
    out = ops.attn_decode(q, cache, block_table=bt, seq_lens=sl, num_q_heads=Hq, num_kv_heads=Hkv, head_dim=D, block_size=bs,
                          scale=D ** -0.5, splits=splits, force_cuda_core=True)
    for r, n in enumerate((300, 17)):
        k, v = (cache[bt[r].long(), i].reshape(-1, Hkv, D)[:n].double().repeat_interleave(Hq // Hkv, 1) for i in (0, 1))
        p = torch.softmax(torch.einsum("hd,khd->hk", q[r].view(Hq, D).double(), k) * D ** -0.5, -1)
        exp = torch.einsum("hk,khd->hd", p, v)
        assert ((out[r].view(Hq, D).double() - exp).norm() / exp.norm()).item() < 2.0 ** -8
    assert ops.read_status() == 0


def test_attn_prefill_of_very_many_tiles():
    """More tiles than a grid's second dimension holds: 66000 requests of one token, each after up to seven others."""
    torch.manual_seed(4)
    D, Hq, Hkv, bs, n = 128, 2, 1, 8, 66000
    cache = _rand(5, 2, bs, Hkv, D)
    bt = (torch.arange(n, device=DEV, dtype=torch.int32) % 5)[:, None].contiguous()
    sl = torch.arange(n, device=DEV, dtype=torch.int32) % bs + 1
    q = _rand(n, Hq * D)
    i32 = dict(device=DEV, dtype=torch.int32)
    out = ops.attn_prefill(q, cache, block_table=bt, seq_lens=sl, q_start=torch.arange(n + 1, **i32), tile_req=torch.arange(n, **i32),
                           tile_q0=torch.zeros(n, **i32), num_q_heads=Hq, num_kv_heads=Hkv, head_dim=D, block_size=bs,
                           scale=D ** -0.5, tile_keys=10 ** 9)
    k, v = (cache[bt[:, 0].long(), i, :, 0].double() for i in (0, 1))
    score = torch.einsum("nhd,nkd->nhk", q.view(n, Hq, D).double(), k) * D ** -0.5
    score = score.masked_fill(torch.arange(bs, device=DEV)[None, None] >= sl[:, None, None], -float("inf"))
    exp = torch.einsum("nhk,nkd->nhd", torch.softmax(score, -1), v).reshape(n, Hq * D)
    assert ((out.double() - exp).norm() / exp.norm()).item() < 2 * 2.0 ** -8
    assert ops.read_status() == 0


def test_attn_prefill_window_softcap():
    torch.manual_seed(10)
    D, Hq, Hkv, bs = 128, 4, 2, 16
    q_lens, ctx = [300, 64], [100, 500]
    seq_lens = [a + b for a, b in zip(q_lens, ctx)]
    cache, bt = _make_paged(seq_lens, Hkv, D, bs)
    T = sum(q_lens)
    q = _rand(T, Hq * D)
    qs = torch.tensor([0, 300, 364], dtype=torch.int32, device=DEV)
    sl = torch.tensor(seq_lens, dtype=torch.int32, device=DEV)
    treq, tq0 = ref.build_prefill_tiles(q_lens)
    kw = dict(block_table=bt, seq_lens=sl, q_start=qs,
              tile_req=torch.tensor(treq, dtype=torch.int32, device=DEV),
              tile_q0=torch.tensor(tq0, dtype=torch.int32, device=DEV), num_q_heads=Hq,
              num_kv_heads=Hkv, head_dim=D, block_size=bs, scale=D ** -0.5)
    out = ops.attn_prefill(q, cache, window=150, softcap=20.0, **kw)
    exp = ref.paged_attention(q, cache, bt, sl, qs, Hq, Hkv, D, bs, D ** -0.5, softcap=20.0,
                              window=150)
    assert _rel_err(out, exp) < 1.5e-2
    assert ops.read_status() == 0


@pytest.mark.parametrize("chunk", [64, 200])
def test_attn_chunked_local(chunk):
    """Chunked-local attention (window < 0): a query sees the keys of its own chunk only, in the
    prefill kernel, the tcgen05 decode kernel and the CUDA-core decode kernel."""
    torch.manual_seed(12)
    D, Hq, Hkv, bs = 128, 8, 2, 16
    q_lens, ctx = [300, 64, 5], [100, 500, 0]
    seq_lens = [a + b for a, b in zip(q_lens, ctx)]
    cache, bt = _make_paged(seq_lens, Hkv, D, bs)
    T = sum(q_lens)
    q = _rand(T, Hq * D)
    qs = torch.tensor([0, 300, 364, 369], dtype=torch.int32, device=DEV)
    sl = torch.tensor(seq_lens, dtype=torch.int32, device=DEV)
    treq, tq0 = ref.build_prefill_tiles(q_lens)
    out = ops.attn_prefill(q, cache, block_table=bt, seq_lens=sl, q_start=qs,
                           tile_req=torch.tensor(treq, dtype=torch.int32, device=DEV),
                           tile_q0=torch.tensor(tq0, dtype=torch.int32, device=DEV), num_q_heads=Hq,
                           num_kv_heads=Hkv, head_dim=D, block_size=bs, scale=D ** -0.5, window=-chunk)
    exp = ref.paged_attention(q, cache, bt, sl, qs, Hq, Hkv, D, bs, D ** -0.5, window=-chunk)
    assert _rel_err(out, exp) < 1.5e-2
    # decode: one query per sequence at its last position
    B = len(seq_lens)
    qd = _rand(B, Hq * D)
    qsd = torch.arange(B + 1, dtype=torch.int32, device=DEV)
    expd = ref.paged_attention(qd, cache, bt, sl, qsd, Hq, Hkv, D, bs, D ** -0.5, window=-chunk)
    for cuda_core in (False, True):
        got = ops.attn_decode(qd, cache, block_table=bt, seq_lens=sl, num_q_heads=Hq, num_kv_heads=Hkv,
                              head_dim=D, block_size=bs, scale=D ** -0.5, window=-chunk, splits=2,
                              force_cuda_core=cuda_core)
        assert _rel_err(got, expd) < 1e-2
    assert ops.read_status() == 0


@pytest.mark.parametrize("D,Hq,Hkv,bs,splits", [(128, 32, 8, 16, 0), (128, 4, 1, 16, 1),
                                                (128, 32, 4, 32, 5), (64, 8, 8, 16, 3),
                                                (256, 24, 4, 16, 2), (128, 16, 8, 16, 4)])
def test_attn_decode(D, Hq, Hkv, bs, splits):
    torch.manual_seed(11)
    seq_lens = [1, 15, 16, 17, 700, 1234, 129]
    cache, bt = _make_paged(seq_lens, Hkv, D, bs)
    B = len(seq_lens)
    q = _rand(B, Hq * D)
    sl = torch.tensor(seq_lens, dtype=torch.int32, device=DEV)
    qs = torch.arange(B + 1, dtype=torch.int32, device=DEV)
    out = ops.attn_decode(q, cache, block_table=bt, seq_lens=sl, num_q_heads=Hq, num_kv_heads=Hkv,
                          head_dim=D, block_size=bs, scale=D ** -0.5, splits=splits)
    exp = ref.paged_attention(q, cache, bt, sl, qs, Hq, Hkv, D, bs, D ** -0.5)
    assert _rel_err(out, exp) < 1e-2
    out2 = ops.attn_decode(q, cache, block_table=bt, seq_lens=sl, num_q_heads=Hq, num_kv_heads=Hkv,
                           head_dim=D, block_size=bs, scale=D ** -0.5, splits=splits, window=100,
                           softcap=30.0)
    exp2 = ref.paged_attention(q, cache, bt, sl, qs, Hq, Hkv, D, bs, D ** -0.5, window=100,
                               softcap=30.0)
    assert _rel_err(out2, exp2) < 1e-2


@pytest.mark.parametrize("Hq,Hkv,bs,splits", [(32, 8, 32, 1), (16, 4, 16, 3)])
def test_attn_decode_tcgen05_persistent(Hq, Hkv, bs, splits):
    """More (sequence, kv head, split) items than resident CTAs: every CTA walks several items
    (some of them empty) and the rings run across the item boundaries."""
    torch.manual_seed(22)
    D = 128
    B = 100 if Hkv == 8 else 60
    gen = torch.Generator().manual_seed(5)
    seq_lens = torch.randint(0, 600, (B,), generator=gen).tolist()
    seq_lens[3] = 0
    seq_lens[7] = 128
    seq_lens[11] = 1
    cache, bt = _make_paged([max(s, 1) for s in seq_lens], Hkv, D, bs)
    q = _rand(B, Hq * D)
    sl = torch.tensor(seq_lens, dtype=torch.int32, device=DEV)
    qs = torch.arange(B + 1, dtype=torch.int32, device=DEV)
    kw = dict(block_table=bt, seq_lens=sl, num_q_heads=Hq, num_kv_heads=Hkv, head_dim=D,
              block_size=bs, scale=D ** -0.5, splits=splits)
    exp = ref.paged_attention(q, cache, bt, sl, qs, Hq, Hkv, D, bs, D ** -0.5)
    for _ in range(2):
        out = ops.attn_decode(q, cache, **kw)
        assert ops.read_status() == 0
        assert _rel_err(out, exp) < 1e-2


@pytest.mark.parametrize("D", [128, 256])
@pytest.mark.parametrize("Hq,Hkv,bs,splits", [(32, 8, 16, 0), (4, 1, 32, 1), (32, 4, 16, 3),
                                              (16, 16, 64, 2), (8, 1, 128, 4), (16, 1, 16, 2),
                                              (24, 4, 32, 2)])
def test_attn_decode_tcgen05(Hq, Hkv, bs, splits, D):
    """tcgen05 swapped-operand decode kernel (head_dim 128 and 256) vs the fp32 oracle and vs the
    CUDA-core kernel."""
    torch.manual_seed(21)
    seq_lens = [1, 127, 128, 129, 700, 1234, 0, 31]
    lens_for_cache = [max(s, 1) for s in seq_lens]
    cache, bt = _make_paged(lens_for_cache, Hkv, D, bs)
    B = len(seq_lens)
    q = _rand(B, Hq * D)
    # strided q like the model passes it (a column slice of the merged qkv buffer)
    wide = _rand(B, (Hq + 2 * Hkv) * D)
    wide[:, : Hq * D] = q
    qv = wide[:, : Hq * D]
    sl = torch.tensor(seq_lens, dtype=torch.int32, device=DEV)
    qs = torch.arange(B + 1, dtype=torch.int32, device=DEV)
    kw = dict(block_table=bt, seq_lens=sl, num_q_heads=Hq, num_kv_heads=Hkv, head_dim=D,
              block_size=bs, scale=D ** -0.5, splits=splits)
    out = ops.attn_decode(qv, cache, **kw)
    assert ops.read_status() == 0
    exp = ref.paged_attention(q, cache, bt, sl, qs, Hq, Hkv, D, bs, D ** -0.5)
    assert _rel_err(out, exp) < 1e-2
    old = ops.attn_decode(qv, cache, force_cuda_core=True, **kw)
    assert _rel_err(out, old) < 1e-2
    out2 = ops.attn_decode(qv, cache, window=100, softcap=30.0, **kw)
    exp2 = ref.paged_attention(q, cache, bt, sl, qs, Hq, Hkv, D, bs, D ** -0.5, window=100,
                               softcap=30.0)
    assert _rel_err(out2, exp2) < 1e-2
    assert ops.read_status() == 0


def test_merge_attn_states():
    torch.manual_seed(12)
    T, H, D = 9, 4, 128
    a, b = _rand(T, H, D), _rand(T, H, D)
    la = torch.randn(T, H, device=DEV)
    lb = torch.randn(T, H, device=DEV)
    lb[0, 0] = -math.inf
    lo = torch.empty_like(la)
    out = ops.merge_attn_states(a, la, b, lb, lse_out=lo)
    mx = torch.maximum(la, lb)
    wa, wb = torch.exp(la - mx), torch.exp(lb - mx)
    exp = (a.float() * wa[..., None] + b.float() * wb[..., None]) / (wa + wb)[..., None]
    assert _rel_err(out, exp) < 5e-3
    assert torch.allclose(lo, mx + torch.log(wa + wb), atol=1e-4)


# ------------------------------------------------------------------------------- sampling
def test_argmax_tie_break_lowest_index():
    torch.manual_seed(13)
    logits = torch.randn(37, 151936, device=DEV)
    logits[3, 100] = 50.0
    logits[3, 90000] = 50.0
    got = ops.argmax(logits)
    assert torch.equal(got, logits.argmax(-1)) or got[3].item() == 100
    assert got[3].item() == 100
    mask = torch.ones(37, dtype=torch.bool)
    mask[3] = False
    assert torch.equal(got[mask], logits.argmax(-1)[mask])


def test_top_k_top_p_min_p_temperature():
    torch.manual_seed(14)
    n, V = 6, 32000
    logits = torch.randn(n, V, device=DEV) * 3
    k = torch.tensor([0, 1, 50, 0, 20, V], dtype=torch.int32, device=DEV)
    p = torch.tensor([1.0, 1.0, 1.0, 0.9, 0.5, 0.3], dtype=torch.float32, device=DEV)
    got = ops.apply_top_k_top_p(logits.clone(), k, p)
    exp = ref.top_k_top_p(logits, k.tolist(), p.tolist())
    assert torch.equal(torch.isinf(got), torch.isinf(exp))
    temp = torch.tensor([0.0, 0.5, 1.0, 2.0, 0.7, 1e-6], device=DEV)
    t = ops.apply_temperature(logits.clone(), temp)
    e = logits.clone()
    for r in range(n):
        if temp[r] >= 1e-5:
            e[r] /= temp[r]
    assert torch.allclose(t, e, rtol=1e-6)
    mp = torch.tensor([0.0, 0.1, 0.5, 0.01, 0.0, 0.2], device=DEV)
    g = ops.apply_min_p(logits.clone(), mp)
    pr = torch.softmax(logits, -1)
    keep = pr >= mp[:, None] * pr.max(-1, keepdim=True).values
    # boundary elements may differ by rounding: compare away from the threshold
    far = (pr / pr.max(-1, keepdim=True).values - mp[:, None]).abs() > 1e-6
    assert torch.equal((~torch.isinf(g))[far], keep[far])


def test_softmax_random_sample_rank():
    torch.manual_seed(15)
    n, V = 4, 5000
    logits = torch.randn(n, V, device=DEV)
    pr = ops.softmax(logits)
    assert torch.allclose(pr, torch.softmax(logits, -1), atol=1e-7, rtol=1e-4)
    lp = ops.softmax(logits, log=True)
    assert torch.allclose(lp, torch.log_softmax(logits, -1), atol=1e-4)
    seeds = torch.tensor([1, 2, 3, 1], dtype=torch.int64, device=DEV).view(torch.int64)
    steps = torch.tensor([0, 0, 5, 0], dtype=torch.int64, device=DEV)
    pr[3] = pr[0]
    s1 = ops.random_sample(pr, seeds, steps)
    s2 = ops.random_sample(pr, seeds, steps)
    assert torch.equal(s1, s2)
    assert s1[0] == s1[3]
    assert ref.race_sample(pr[0].cpu(), 1, 0) == s1[0].item()
    assert ref.race_sample(pr[2].cpu(), 3, 5) == s1[2].item()
    # distribution sanity: many steps on a peaked 4-token row
    probs = torch.zeros(2000, 8, device=DEV)
    probs[:, :4] = torch.tensor([0.5, 0.25, 0.125, 0.125], device=DEV)
    sd = torch.full((2000,), 42, dtype=torch.int64, device=DEV)
    st = torch.arange(2000, dtype=torch.int64, device=DEV)
    draws = ops.random_sample(probs, sd, st)
    freq = torch.bincount(draws, minlength=8).float() / 2000
    assert abs(freq[0].item() - 0.5) < 0.05 and abs(freq[1].item() - 0.25) < 0.05
    toks = torch.tensor([5, 6, 7, 8], device=DEV)
    tl, rk = ops.token_rank(lp, toks)
    assert torch.allclose(tl, lp[torch.arange(n), toks])
    exp_rank = (lp > lp[torch.arange(n), toks][:, None]).sum(-1) + 1
    assert torch.equal(rk.long(), exp_rank)


def test_penalties_bias_mask_bitmask():
    torch.manual_seed(16)
    n, V = 3, 1000
    logits = torch.randn(n, V, device=DEV)
    rows = torch.tensor([0, 0, 2], dtype=torch.int32, device=DEV)
    toks = torch.tensor([5, 9, 7], dtype=torch.int32, device=DEV)
    cnt = torch.tensor([2, 0, 1], dtype=torch.int32, device=DEV)
    rep = torch.tensor([1.5, 1.0, 2.0], device=DEV)
    freq = torch.tensor([0.1, 0.0, 0.2], device=DEV)
    pres = torch.tensor([0.3, 0.0, 0.4], device=DEV)
    got = ops.apply_penalties(logits.clone(), rows, toks, cnt, rep, freq, pres)
    exp = logits.clone()
    for r, t, c in zip(rows.tolist(), toks.tolist(), cnt.tolist()):
        v = exp[r, t]
        v = v / rep[r] if v > 0 else v * rep[r]
        v = v - freq[r] * c - (pres[r] if c > 0 else 0.0)
        exp[r, t] = v
    assert torch.allclose(got, exp, atol=1e-6)
    vals = torch.tensor([1.0, -2.0, 3.0], device=DEV)
    got = ops.apply_logit_bias(logits.clone(), rows, toks, vals)
    exp = logits.clone()
    exp[rows.long(), toks.long()] += vals
    assert torch.allclose(got, exp)
    got = ops.apply_token_mask(logits.clone(), rows, toks)
    assert torch.isinf(got[0, 5]) and torch.isinf(got[2, 7]) and not torch.isinf(got[1]).any()
    words = (V + 31) // 32
    mask = torch.randint(-2**31, 2**31 - 1, (2, words), dtype=torch.int32, device=DEV)
    row_ids = torch.tensor([2, 0], dtype=torch.int32, device=DEV)
    got = ops.apply_bitmask(logits.clone(), mask, row_ids)
    bits = ((mask[:, :, None] >> torch.arange(32, device=DEV)) & 1).reshape(2, -1)[:, :V].bool()
    assert torch.equal(~torch.isinf(got[2]), bits[0])
    assert torch.equal(~torch.isinf(got[0]), bits[1])
    assert not torch.isinf(got[1]).any()


def test_greedy_rejection():
    draft = torch.tensor([5, 6, 7, 1, 2], device=DEV)
    cu = torch.tensor([0, 3, 5], dtype=torch.int32, device=DEV)
    # request 0: 3 drafts + bonus -> rows 0..3 ; request 1: 2 drafts + bonus -> rows 4..6
    target = torch.tensor([5, 6, 9, 11, 1, 2, 13], device=DEV)
    out = ops.greedy_reject(target, draft, cu, 3)
    assert out.tolist() == [[5, 6, 9, -1], [1, 2, 13, -1]]


@pytest.mark.parametrize("M,I,K,kind", [(1280, 1024, 512, 0), (300, 384, 256, 1), (64, 256, 128, 0), (200, 14336, 4096, 0),
                                        (700, 14336, 4096, 0), (2048, 128, 64, 2)])
def test_gemm_gated_activation(M, I, K, kind):
    """act(gate) * up in the GEMM epilogue (interleaved gate / up rows). With the same tiling and
    no stream-K split it equals the bf16 GEMM followed by the activation kernel bit for bit;
    otherwise (fp32 partial sums added in another order) within bf16 rounding."""
    torch.manual_seed(3)
    a = _rand(M, K)
    wg, wu = _rand(I, K, scale=0.05), _rand(I, K, scale=0.05)
    w_il = ops.interleave_gate_up(wg, wu)
    merged_w = torch.cat([wg, wu], 0)
    exp = ref.act_and_mul(ref.gemm(a, merged_w), kind)
    out = ops.gemm_gated(a, w_il, kind)
    assert ops.read_status() == 0
    assert _rel_err(out, exp) < 2e-2
    if M > 128:
        two_step = ops.act_and_mul(ops.gemm(a, merged_w, force_path=7), kind)
        assert torch.equal(ops.gemm_gated(a, w_il, kind, force_path=7), two_step)
        assert _rel_err(ops.gemm_gated(a, w_il, kind, force_path=9), exp) < 2e-2
    else:
        assert torch.equal(out, ops.act_and_mul(ops.gemm(a, merged_w), kind))


@pytest.mark.parametrize("V,ld", [(5, 8), (37, 37), (1003, 1003), (32000, 32000), (151936, 151936), (420001, 420004)])
def test_row_kernels_over_a_cluster(V, ld):
    """Rows shared by the CTAs of a cluster: slices of no, few and many columns, unaligned rows, rows too long for shared
    memory. The threshold of top-p may move by one logit where the mass is within 1e-5 of p (order of the sums)."""
    torch.manual_seed(V)
    n = 6
    x = torch.randn(n, ld, device=DEV)[:, :V] * 2
    x[1, V // 2:] = -float("inf")
    k = torch.tensor([0, min(3, V), min(50, V), 1, V, min(7, V)], dtype=torch.int32, device=DEV)
    p = torch.tensor([0.9, 1.0, 0.95, 0.5, 0.3, 1.0], device=DEV)
    got = torch.empty(n, ld, device=DEV)[:, :V]
    got.copy_(x)
    ops.apply_top_k_top_p(got, k, p)
    for r in range(n):
        srt = x[r].double().sort(descending=True).values
        keep = V if k[r] <= 0 or k[r] >= V else int(k[r])
        if p[r] < 1:
            mass = torch.softmax(srt[:keep], 0).cumsum(0)
            least, most = (min(int((mass < float(p[r]) + d).sum()), keep - 1) + 1 for d in (-1e-5, 1e-5))
        else:
            least = most = keep
        kept = torch.isfinite(got[r])
        n_kept = int(kept.sum())
        assert least <= n_kept <= most or n_kept == int(torch.isfinite(x[r]).sum()) < least
        assert not n_kept or bool((x[r][kept].min() > x[r][~kept]).all())      # the largest ones
        assert torch.equal(got[r][kept], x[r][kept])
    soft = ops.softmax(x)
    exact = torch.softmax(x.double(), -1)
    assert ((soft.double() - exact).norm() / exact.norm()).item() < 2e-6 + 4e-7 * float(x[torch.isfinite(x)].abs().max())
    logp = ops.softmax(x, log=True)
    fin = torch.isfinite(x)
    assert (logp.double() - torch.log_softmax(x.double(), -1))[fin].abs().max().item() < 2e-5
    seeds = torch.arange(n, dtype=torch.int64, device=DEV) + 11
    steps = torch.full((n,), 3, dtype=torch.int64, device=DEV)
    tok = ops.random_sample(torch.softmax(got, -1).contiguous(), seeds, steps)
    again = ops.random_sample(torch.softmax(got, -1).contiguous(), seeds, steps)
    assert torch.equal(tok, again) and all(torch.isfinite(got[r, tok[r]]) for r in range(n))
    assert ops.read_status() == 0


@pytest.mark.parametrize("V", [9021, 20000])
def test_rows_of_one_and_of_eight_ctas(V):
    """Six rows of V columns take a cluster of eight CTAs each, 160 copies of them (more rows than SMs) one CTA each. Top-k,
    top-p away from a tie of the mass, ties and infinities at the threshold, and the draw from the same probabilities: the
    same bits; softmax: sums in another order."""
    torch.manual_seed(V)
    inf = float("inf")
    x = torch.randn(6, V, device=DEV) * 2
    x[1, 4:] = -inf                                       # fewer finite logits than k: the threshold is -inf
    x[2] = x[2].round()                                   # many ties at the threshold: all are kept
    x[3, 17] = inf                                        # its mass is not a number: top-k alone decides
    x[4] = -inf
    x[4, V - 1] = 3.0
    k = torch.tensor([50, 10, 20, 8, 5, 0], dtype=torch.int32, device=DEV)
    p = torch.tensor([1.0, 1.0, 1.0, 0.9, 0.9, 0.8], device=DEV)
    many = [t.repeat(27, *([1] * (t.dim() - 1)))[:160].contiguous() for t in (x, k, p)]
    few, lots = x.clone(), many[0].clone()
    ops.apply_top_k_top_p(few, k, p)
    ops.apply_top_k_top_p(lots, many[1], many[2])
    rows = torch.arange(160, device=DEV) % 6
    assert torch.equal(few[rows], lots)
    kept = (few == x) & (x > -inf)
    assert int(kept[0].sum()) == 50 and torch.equal(few[1], x[1]) and torch.equal(few[4], x[4])
    kth = x[2].sort(descending=True).values[19]
    assert torch.equal(kept[2], x[2] >= kth)
    assert int(kept[3].sum()) == 8 and bool(kept[3, 17])
    mass = torch.softmax(x[5].double(), 0).sort(descending=True).values.cumsum(0)
    assert abs(int(kept[5].sum()) - int((mass < 0.8).sum()) - 1) <= 1
    soft = [ops.softmax(t[[0, 2, 5]] if t.shape[0] == 6 else t) for t in (few, lots)]
    assert (soft[0] - soft[1][[0, 2, 5]]).abs().max().item() < 1e-6
    probs = torch.softmax(few[[0, 2, 5]], -1)
    seeds = torch.arange(3, dtype=torch.int64, device=DEV) + 5
    big = [t.repeat(54, *([1] * (t.dim() - 1)))[:160].contiguous() for t in (probs, seeds)]
    steps = torch.full((160,), 9, dtype=torch.int64, device=DEV)
    assert torch.equal(ops.random_sample(probs, seeds, steps[:3])[torch.arange(160, device=DEV) % 3], ops.random_sample(*big, steps))
    assert ops.read_status() == 0


@pytest.mark.parametrize("H", [8, 264, 2040, 2048, 2056, 4096, 4104, 8192, 8200])
def test_rmsnorm_of_every_number_of_vectors_a_thread(H):
    """One, two, four vectors a thread in registers or, beyond 8192, a loop through shared memory; the last one partly
    empty; results in place of the input."""
    torch.manual_seed(H)
    for T in (1, 3):
        x, w, r = _rand(T, H), _rand(H), _rand(T, H)
        exp, newr = ref.rmsnorm(x, w, 1e-6, residual=r)
        r2, x2 = r.clone(), x.clone()
        ops.rmsnorm(x2, w, 1e-6, residual=r2, out=x2)
        assert torch.equal(r2, newr)
        assert _rel_err(x2, exp) < 2.0 ** -8                    # (one rounding to bf16)


@pytest.mark.parametrize("Hq,Hkv,T,pad,qk_norm", [(32, 8, 103, 0, False), (5, 3, 600, 0, True), (4, 1, 900, 4, True),
                                                  (7, 1, 1100, 8, False), (16, 8, 129, 0, True)])
def test_rope_kv_of_many_tokens(Hq, Hkv, T, pad, qk_norm):
    """Eight heads a warp: groups that end in k or v heads or in none, rows with a pitch that only 8-byte pieces read, tokens
    without a slot, q to a tensor of its own."""
    torch.manual_seed(T)
    D, bs = 128, 16
    nb = T // bs + 1
    ld = (Hq + 2 * Hkv) * D + pad
    rows = _rand(T, ld)
    qkv = rows[:, : ld - pad]
    pos = torch.randint(0, 500, (T,), device=DEV)
    table = ops.rope_table(ref.rope_inv_freq(D, 1e6).to(DEV), 512)
    qn, kn = (_rand(D), _rand(D)) if qk_norm else (None, None)
    slots = torch.randperm(nb * bs, device=DEV)[:T].to(torch.int64)
    slots[5] = -1
    eq, ek, ev = ref.rope_kv(qkv.contiguous(), pos, table, Hq, Hkv, D, D, True, qn, kn)
    exp = torch.zeros(nb, 2, bs, Hkv, D, device=DEV, dtype=torch.bfloat16)
    ref.write_kv_cache(exp, ek, ev, slots, bs)
    for own in (False, True):
        work, cache = rows.clone()[:, : ld - pad], torch.zeros_like(exp)
        q_out = torch.empty(T, Hq * D, device=DEV, dtype=torch.bfloat16) if own else None
        ops.rope_kv(work, pos, table, num_q_heads=Hq, num_kv_heads=Hkv, head_dim=D, rot_dim=D, q_norm=qn, k_norm=kn,
                    slot_mapping=slots, kv_cache=cache, block_size=bs, q_out=q_out)
        got = q_out if own else work[:, : Hq * D]
        assert _rel_err(got.reshape(T, Hq, D), eq) < 8e-3
        assert _rel_err(cache[:, 0], exp[:, 0]) < 8e-3
        assert torch.equal(cache[:, 1], exp[:, 1])
        if own:
            assert torch.equal(work[:, : Hq * D], qkv[:, : Hq * D])


@pytest.mark.parametrize("T,Hq,Hkv,H,qk_norm,fp8", [(3, 4, 1, 256, True, False), (16, 32, 8, 1024, False, False), (45, 5, 3, 264, True, False),
                                                    (128, 16, 8, 512, True, False), (1, 6, 2, 256, False, True), (33, 8, 2, 1024, True, True)])
def test_qkv_product_with_rotation(T, Hq, Hkv, H, qk_norm, fp8):
    """The attention half of a block does qk-norm, rotation and cache write in the product's epilogue: the bits of the three
    kernels one after the other."""
    from vllm_cpp_b200.ops import quant as Q
    from vllm_cpp_b200.ops.layer import DenseLayerWeights, DenseStep, dense_attn_half
    torch.manual_seed(T + H)
    D, bs = 128, 16
    N, nb = (Hq + 2 * Hkv) * D, T // bs + 2
    hidden, ln1, wo = _rand(T, H), _rand(H), _rand(H, Hq * D, scale=0.05)
    wqkv = _rand(N, H, scale=0.05)
    qn, kn = (_rand(D), _rand(D)) if qk_norm else (None, None)
    pos = torch.randint(0, 500, (T,), device=DEV)
    slots = torch.randperm(nb * bs, device=DEV)[:T].to(torch.int64)
    slots[T // 2] = -1
    table = ops.rope_table(ref.rope_inv_freq(D, 1e6).to(DEV), 512)
    cache, exp = (torch.zeros(nb, 2, bs, Hkv, D, device=DEV, dtype=torch.bfloat16) for _ in range(2))
    w, s = DenseLayerWeights(), DenseStep()
    keep = [torch.empty(T, max(H, Hq * D), device=DEV, dtype=torch.uint8), torch.empty(T, device=DEV)]
    if fp8:
        scales = torch.rand(N, device=DEV) * 0.01
        w8, o8 = wqkv.clamp(-1, 1).to(torch.float8_e4m3fn), wo.to(torch.float8_e4m3fn)
        so = torch.ones(H, device=DEV)
        w.fp8, w.qkv, w.o, w.qkv_scale, w.o_scale = 1, w8.data_ptr(), o8.data_ptr(), scales.data_ptr(), so.data_ptr()
        s.fp8_act, s.fp8_scales = keep[0].data_ptr(), keep[1].data_ptr()
        a8, sa = Q.quant_fp8_rowwise(hidden, norm_weight=ln1)
        want = Q.gemm_fp8(a8, w8, sa, scales)
    else:
        w.qkv, w.o = wqkv.data_ptr(), wo.data_ptr()
        want = ops.gemm(ops.rmsnorm(hidden, ln1, 1e-6), wqkv)
    ops.rope_kv(want, pos, table, num_q_heads=Hq, num_kv_heads=Hkv, head_dim=D, rot_dim=D, q_norm=qn, k_norm=kn,
                slot_mapping=slots, kv_cache=exp, block_size=bs)
    qkv, attn, resid, normed = (torch.zeros(T, n, device=DEV, dtype=torch.bfloat16) for n in (N, Hq * D, H, H))
    w.ln1, w.kv_cache = ln1.data_ptr(), cache.data_ptr()
    w.q_norm, w.k_norm = (t.data_ptr() if t is not None else None for t in (qn, kn))
    s.T, s.H, s.Hq, s.Hkv, s.D, s.rot, s.block_size, s.neox, s.eps, s.num_blocks = T, H, Hq, Hkv, D, D, bs, 1, 1e-6, nb
    s.positions, s.cos_sin, s.slot_mapping, s.first_layer = pos.data_ptr(), table.data_ptr(), slots.data_ptr(), 1
    s.hidden, s.resid, s.normed, s.qkv_buf, s.attn = (t.data_ptr() for t in (hidden, resid, normed, qkv, attn))
    ws = ops.workspace(torch.device(DEV), ops.GEMM_WS_BYTES)
    s.gemm_ws, s.gemm_ws_bytes = ws.data_ptr(), ws.numel()
    dense_attn_half(w, s)
    assert torch.equal(qkv, want)
    assert torch.equal(cache, exp)
    assert ops.read_status() == 0


@pytest.mark.parametrize("T,H,I", [(300, 256, 384), (257, 512, 128)])
def test_fp8_block_with_and_without_a_buffer_for_the_activation(T, H, I):
    """From 257 rows on act(gate) * up goes to ``act`` where there is one at a multiple of 16 bytes, else through ``gate_up_buf``: the same bits."""
    from vllm_cpp_b200.ops.layer import DenseLayerWeights, DenseStep, dense_layer
    torch.manual_seed(T)
    D, Hq, Hkv, bs = 128, 2, 1, 16
    N, nb = (Hq + 2 * Hkv) * D, T // bs + 2
    hidden0, ln1, ln2 = _rand(T, H), _rand(H), _rand(H)
    w, s = DenseLayerWeights(), DenseStep()
    mats = {k: _rand(*shape).clamp(-1, 1).to(torch.float8_e4m3fn) for k, shape in
            (("qkv", (N, H)), ("o", (H, Hq * D)), ("gate_up", (2 * I, H)), ("down", (H, I)))}
    scales = {k: torch.rand(m.shape[0], device=DEV) * 0.01 for k, m in mats.items()}
    cache = torch.zeros(nb, 2, bs, Hkv, D, device=DEV, dtype=torch.bfloat16)
    for k, m in mats.items():
        setattr(w, k, m.data_ptr())
        setattr(w, k + "_scale", scales[k].data_ptr())
    w.fp8, w.ln1, w.ln2, w.kv_cache = 1, ln1.data_ptr(), ln2.data_ptr(), cache.data_ptr()
    pos, slots = torch.arange(T, device=DEV), torch.arange(T, device=DEV)
    table = ops.rope_table(ref.rope_inv_freq(D, 1e6).to(DEV), 512)
    resid, normed, qkv, gate_up = (torch.zeros(T, n, device=DEV, dtype=torch.bfloat16) for n in (H, H, N, 2 * I))
    room, attn = torch.zeros(T * I + 8, device=DEV, dtype=torch.bfloat16), _rand(T, Hq * D)       # (no request: attn stays as it is)
    act8, row_scales = torch.empty(T, max(H, Hq * D, I), device=DEV, dtype=torch.uint8), torch.empty(T, device=DEV)
    ws = ops.workspace(torch.device(DEV), ops.GEMM_WS_BYTES)
    s.T, s.H, s.Hq, s.Hkv, s.D, s.rot, s.inter, s.block_size, s.neox, s.eps, s.num_blocks = T, H, Hq, Hkv, D, D, I, bs, 1, 1e-6, nb
    s.gate_up_interleaved, s.first_layer = 1, 1
    s.positions, s.cos_sin, s.slot_mapping = pos.data_ptr(), table.data_ptr(), slots.data_ptr()
    s.resid, s.normed, s.qkv_buf, s.attn, s.gate_up_buf = (t.data_ptr() for t in (resid, normed, qkv, attn, gate_up))
    s.fp8_act, s.fp8_scales, s.gemm_ws, s.gemm_ws_bytes = act8.data_ptr(), row_scales.data_ptr(), ws.data_ptr(), ws.numel()
    got = []
    for at in (room.data_ptr(), room.data_ptr() + 8, None):
        hidden = hidden0.clone()
        s.hidden, s.act = hidden.data_ptr(), at
        dense_layer(w, s)
        got.append(hidden)
    assert ops.read_status() == 0
    assert torch.isfinite(got[0]).all() and float(got[0].float().abs().max()) > 0
    assert torch.equal(got[0], got[1]) and torch.equal(got[0], got[2])


@pytest.mark.parametrize("M,N,K", [(130, 1024, 1040), (257, 384, 4096), (300, 512, 1288), (129, 128, 8192), (513, 256, 2048)])
@pytest.mark.parametrize("path", [5, 6, 9, 10])
def test_gemm_tiles_in_parts(M, N, K, path):
    """Few tiles: every one is shared by equal parts of K, two to eight of them, also where neither K nor the columns divide;
    twice on the same counters, with what follows the product. fp32 sums of exact products, rounded to bf16 once (2^-8)."""
    torch.manual_seed(M + N)
    a, w, bias, res = _rand(M, K), _rand(N, K, scale=K ** -0.5), _rand(N), _rand(M, N)
    exp = a.double() @ w.double().t()
    first = ops.gemm(a, w, force_path=path)
    assert _rel_err(first.double(), exp) < 2.0 ** -8
    assert torch.equal(first, ops.gemm(a, w, force_path=path))
    out = torch.full((M, N), 7.0, device=DEV, dtype=torch.float32)
    ops.gemm(a, w, bias=bias, residual=res, out=out, force_path=path)
    assert _rel_err(out.double(), exp + bias.double() + res.double()) < 1e-5
    if path == 9 and N % 256 == 0:
        got = ops.gemm_gated(a, ops.interleave_gate_up(w[: N // 2], w[N // 2:]), force_path=9)
        g, u = exp[:, : N // 2], exp[:, N // 2:]
        assert _rel_err(got.double(), g * torch.sigmoid(g) * u) < 2.0 ** -6     # (three roundings)
    assert ops.read_status() == 0


@pytest.mark.parametrize("M,N,K", [(129, 8, 64), (200, 136, 328), (260, 128, 72), (300, 200, 1024), (1100, 264, 520), (2000, 3072, 768)])
def test_gemm_of_the_form_that_is_chosen(M, N, K):
    """Narrow and ragged matrices through the estimate, against 64 bits."""
    torch.manual_seed(M)
    a, w = _rand(M, K), _rand(N, K, scale=K ** -0.5)
    assert _rel_err(ops.gemm(a, w).double(), a.double() @ w.double().t()) < 2.0 ** -8
    assert ops.read_status() == 0


@pytest.mark.parametrize("N,K,first,form", [(16376, 1024, 129, 0), (16384, 2048, 49, 6), (18432, 1024, 49, 6), (28672, 4096, 65, 5),
                                            (57344, 1024, 64, 6), (57344, 512, 17, 5), (128256, 4096, 33, 5), (151936, 1024, 49, 5)])
def test_form_of_few_rows_of_wide_matrices(N, K, first, form):
    """Where the line between a cluster and the tiles lies (148 SMs), and which tiles follow; both sides give the product."""
    from vllm_cpp_b200.ops import _lib
    forms = [_lib.lib().b200_gemm_form(m, N, K) for m in range(1, 129)]
    assert not any(forms[: first - 1]) and forms[first - 1: first] in ([form], []) and all(forms[first - 1:])
    if N > 65536:
        return
    torch.manual_seed(N)
    w = _rand(N, K, scale=K ** -0.5)
    for M in (first - 1, first):
        a = _rand(M, K)
        assert _rel_err(ops.gemm(a, w), a.float() @ w.float().t()) < 2.0 ** -8
    assert ops.read_status() == 0


@pytest.mark.parametrize("V,n", [(1024, 5), (3000, 5), (151936, 5), (9021, 160)])
def test_top_k_of_about_what_a_list_holds(V, n):
    """The search goes on in a list once 1024 values of the row are left: k below, at and above that, ties that do not fit,
    unaligned rows, one and eight CTAs a row; then top-p among them, with a threshold that the sums' order cannot move."""
    torch.manual_seed(V + n)
    x = torch.randn(n, V + 3, device=DEV)[:, :V] * 3
    x[2] = (x[2] * 2).round()                              # hundreds of ties at every value
    ks = [min(k, V - 1) for k in (50, 1023, 1024, 1025, 700)]
    k = torch.tensor([ks[r % 5] for r in range(n)], dtype=torch.int32, device=DEV)
    got = x.clone()
    ops.apply_top_k_top_p(got, k, None)
    for r in range(n):
        kth = x[r].topk(int(k[r])).values[-1]
        assert torch.equal(got[r], torch.where(x[r] >= kth, x[r], -float("inf")))
    # half of the mass: far from a value of the cumulative sum where the values are distinct
    half = x.clone()
    ops.apply_top_k_top_p(half, k, torch.full((n,), 0.5, device=DEV))
    for r in (0, 1, 3, 4):
        srt = got[r].double().sort(descending=True).values[: int(k[r])]
        mass = torch.softmax(srt, 0).cumsum(0)
        least, most = (int((mass < 0.5 + d).sum()) + 1 for d in (-1e-5, 1e-5))
        assert least <= int(torch.isfinite(half[r]).sum()) <= most
    assert ops.read_status() == 0


@pytest.mark.parametrize("B,Hkv", [(37, 8), (38, 8), (75, 4)])
def test_attn_decode_of_two_and_of_three_ctas_an_sm(B, Hkv):
    """Grids of 296 CTAs and of a few more (148 SMs): sequences of none to five tiles, scores that raise the reference maximum late."""
    torch.manual_seed(B)
    Hq, D, bs = Hkv * 4, 128, 16
    lens = [(i * 53) % 600 for i in range(B)]
    lens[1], lens[2], lens[3] = 1, 128, 129
    cache, bt = _make_paged([max(n, 1) for n in lens], Hkv, D, bs)
    cache[:, 0] *= torch.linspace(0.2, 6.0, cache.shape[0], device=DEV)[:, None, None, None].to(torch.bfloat16)
    q = _rand(B, Hq * D)
    sl = torch.tensor(lens, dtype=torch.int32, device=DEV)
    out = ops.attn_decode(q, cache, block_table=bt, seq_lens=sl, num_q_heads=Hq, num_kv_heads=Hkv, head_dim=D, block_size=bs,
                          scale=D ** -0.5, splits=1)
    for b, n in enumerate(lens):
        if n == 0:
            assert not out[b].any()
            continue
        kv = cache[bt[b, : (n + bs - 1) // bs].long()]                       # [blocks, 2, bs, Hkv, D]
        k, v = (kv[:, i].reshape(-1, Hkv, D)[:n].float().repeat_interleave(4, 1) for i in range(2))
        s = torch.einsum("hd,thd->ht", q[b].float().view(Hq, D), k) * D ** -0.5
        exp = torch.einsum("ht,thd->hd", torch.softmax(s, -1), v)
        assert _rel_err(out[b].view(Hq, D), exp) < 8e-3                      # P and the result in bf16
    assert ops.read_status() == 0
