"""MoE kernels (router top-k, expert sort, tcgen05 grouped GEMM, combine) and the Qwen3-MoE
model end to end, against the fp32 PyTorch restatements."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from vllm_cpp_b200 import ops  # noqa: E402
from vllm_cpp_b200.ops import moe as M  # noqa: E402

DEV = "cuda"


def _rel(a, b):
    from _numerics import rel_err
    return rel_err(a, b, row_tol=0.15, abs_tol=0.1)


@pytest.mark.parametrize("T,E,k", [(7, 128, 8), (300, 64, 6), (33, 8, 2)])
def test_router_topk_softmax_renorm(T, E, k):
    torch.manual_seed(0)
    logits = torch.randn(T, E, device=DEV)
    logits[0, 3] = logits[0, 5] = 9.0          # tie: the lower index must win first
    ids, w = M.router_topk(logits, k, renorm=True)
    eids, ew = M.ref_router_topk(logits, k, renorm=True)
    assert torch.equal(ids, eids)
    assert torch.allclose(w, ew, atol=1e-6, rtol=1e-5)
    assert ids[0, 0].item() == 3 and ids[0, 1].item() == 5


@pytest.mark.parametrize("T,E,k", [(1, 1, 1), (5, 33, 33), (3, 64, 40), (9, 256, 8), (4, 257, 8)])
@pytest.mark.parametrize("scoring,biased", [("softmax", False), ("sigmoid", True), ("sigmoid", False)])
def test_router_of_a_warp_and_of_a_block(T, E, k, scoring, biased):
    """A warp per token up to 256 experts, a block beyond; more choices than lanes, expert counts around 32, and rows of
    equal logits (the lower index first)."""
    torch.manual_seed(E)
    logits = torch.randn(T, E, device=DEV)
    logits[-1] = logits[-1].round()
    bias = torch.randn(E, device=DEV) * 0.1 if biased else None
    ids, w = M.router_topk(logits, k, renorm=True, scoring=scoring, e_bias=bias, routed_scale=1.5)
    eids, ew = M.ref_router_topk(logits, k, renorm=True, scoring=scoring, e_bias=bias, routed_scale=1.5)
    assert torch.equal(ids, eids)
    assert torch.allclose(w, ew, atol=1e-6, rtol=1e-5)


def test_router_grouped_sigmoid_bias():
    torch.manual_seed(1)
    T, E, k = 40, 64, 6
    logits = torch.randn(T, E, device=DEV)
    bias = torch.randn(E, device=DEV) * 0.1
    ids, w = M.router_topk(logits, k, renorm=True, scoring="sigmoid", e_bias=bias, n_group=8,
                           topk_group=4, routed_scale=2.5)
    eids, ew = M.ref_router_topk(logits, k, renorm=True, scoring="sigmoid", e_bias=bias,
                                 n_group=8, topk_group=4, routed_scale=2.5)
    assert torch.equal(ids.sort(-1).values, eids.sort(-1).values)
    assert torch.allclose(w.sum(-1), ew.sum(-1), atol=1e-5)


def local_pairs(ids, e0, el):
    return int(((ids >= e0) & (ids < e0 + el)).sum().item())


@pytest.mark.parametrize("T,E,k,H,I,e0,el", [(5, 8, 2, 256, 128, 0, 8), (300, 16, 4, 512, 256, 0, 16),
                                             (700, 8, 2, 256, 128, 4, 4), (64, 128, 8, 2048, 768, 0, 128)])
def test_moe_block_matches_reference(T, E, k, H, I, e0, el):
    """sort + gather + grouped GEMM (gate_up) + silu*mul + grouped GEMM (down) + combine;
    with e0/el a subset of experts is local (expert parallel partial sums)."""
    torch.manual_seed(2)
    x = (torch.randn(T, H, device=DEV) * 0.5).to(torch.bfloat16)
    wgu = (torch.randn(el, 2 * I, H, device=DEV) * 0.05).to(torch.bfloat16)
    wd = (torch.randn(el, H, I, device=DEV) * 0.05).to(torch.bfloat16)
    logits = torch.randn(T, E, device=DEV)
    ids, w = M.router_topk(logits, k)
    ws = M.MoeWorkspace(torch.device(DEV), T, k, el, H, I)
    M.moe_sort(ids, e0, e0 + el, ws)
    P = T * k
    M.moe_gather(x, ws, el, P)
    M.grouped_gemm(ws.xs, wgu, ws.gu, ws, P)
    ops.act_and_mul(ws.gu[:P], 0, out=ws.act[:P])
    # the gated grouped GEMM (both halves in TMEM, activation in the epilogue) gives the same bits
    unfused = ws.act[:local_pairs(ids, e0, el)].clone()
    ws.act.zero_()
    M.grouped_gemm_gated(ws.xs, wgu, ws.act, ws, P, kind=0)
    assert torch.equal(ws.act[:unfused.shape[0]], unfused)
    M.grouped_gemm(ws.act, wd, ws.y, ws, P)
    out = torch.empty(T, H, dtype=torch.bfloat16, device=DEV)
    M.combine(ws.y, ws, w, out)
    exp = M.ref_moe_block(x, ids, w, wgu, wd, e0=e0)
    assert ops.read_status() == 0
    assert _rel(out, exp) < 2e-2
    # bookkeeping: every local pair has a slot, counts add up
    local = ((ids >= e0) & (ids < e0 + el)).sum().item()
    assert ws.meta[2 * el].item() == local
    assert (ws.pair_pos.view(T, k)[(ids >= e0) & (ids < e0 + el)] >= 0).all()


@pytest.mark.parametrize("T,E,H,I,skew", [(1, 64, 72, 136, False), (3, 128, 256, 128, False), (17, 16, 200, 1408, False),
                                          (129, 64, 128, 192, True), (300, 64, 256, 64, True)])
def test_grouped_gemm_of_few_rows_an_expert(T, E, H, I, skew):
    """Weight-bound chunks over a cluster: ragged row tiles and k-blocks, boxes of 16 to 128 rows, more rows than one pass
    takes (``skew``: every token goes to expert 1 too). Each of the two products rounds its values to bf16 (2^-8), the gated
    one three times."""
    torch.manual_seed(T + I)
    x = (torch.randn(T, H, device=DEV)).to(torch.bfloat16)
    wgu = (torch.randn(E, 2 * I, H, device=DEV) * H ** -0.5).to(torch.bfloat16)
    wd = (torch.randn(E, H, I, device=DEV) * I ** -0.5).to(torch.bfloat16)
    ids = torch.stack([torch.randperm(E - 2, device=DEV)[:2] + 2 for _ in range(T)]).int()
    if skew:
        ids[:, 1] = 1
    ws = M.MoeWorkspace(torch.device(DEV), T, 2, E, H, I)
    M.moe_sort(ids, 0, E, ws)
    P = 2 * T
    M.moe_gather(x, ws, E, P)
    ws.act.fill_(7.0)
    M.grouped_gemm_gated(ws.xs, wgu, ws.act, ws, P, kind=1)
    M.grouped_gemm(ws.act, wd, ws.y, ws, P)
    pos, tok = ws.pair_pos.view(T, 2).long(), torch.arange(T, device=DEV)
    for j in range(2):
        e = ids[:, j].long()
        g, u = (torch.einsum("th,tih->ti", x.float(), wgu[e][:, h * I:(h + 1) * I].float()) for h in range(2))
        act = torch.nn.functional.gelu(g, approximate="tanh") * u
        got = ws.act[pos[:, j]].float()
        assert ((got - act).norm() / act.norm()).item() < 3 * 2.0 ** -8
        y = torch.einsum("ti,thi->th", got, wd[e].float())
        assert ((ws.y[pos[:, j]].float() - y).norm() / y.norm()).item() < 2.0 ** -8
    assert bool((ws.act[P:] == 7.0).all())                      # nothing beyond the sorted rows
    assert ops.read_status() == 0


def test_moe_engine_gpu_vs_cpu():
    from vllm_cpp_b200.config import EngineArgs, synthetic_config
    from vllm_cpp_b200.engine import LLM, SamplingParams
    cfg = synthetic_config("tiny-moe")
    cfg.head_dim = 128
    g = torch.Generator().manual_seed(4)
    prompts = [torch.randint(0, cfg.vocab_size, (n,), generator=g).tolist() for n in (90, 7, 200)]
    sp = SamplingParams(temperature=0.0, max_tokens=8, ignore_eos=True)

    def run(dev):
        llm = LLM(EngineArgs(model_config=cfg, device=dev, block_size=16, num_blocks=128,
                             max_model_len=512, max_num_seqs=4, max_num_batched_tokens=256))
        return [o.outputs[0].token_ids for o in llm.generate(prompts, sp)]

    gpu, cpu = run("cuda"), run("cpu")
    assert ops.read_status() == 0
    assert [a[0] for a in gpu] == [a[0] for a in cpu]
    hit = sum(sum(1 for p, q in zip(a, b) if p == q) for a, b in zip(gpu, cpu))
    assert hit / sum(len(a) for a in gpu) > 0.7


@pytest.mark.parametrize("chunks", [3, 40000, 65535])
def test_grouped_gemm_gated_with_a_long_chunk_list(chunks):
    """As many chunks as a grid's second dimension holds, whatever the parts that a chunk is taken in; those past the count on
    the device are nothing."""
    torch.manual_seed(1)
    T, H, I = 300, 64, 136
    x = torch.randn(T, H, device=DEV).to(torch.bfloat16)
    wgu = (torch.randn(1, 2 * I, H, device=DEV) * H ** -0.5).to(torch.bfloat16)
    ws = M.MoeWorkspace(torch.device(DEV), T, 1, 1, H, I)
    M.moe_sort(torch.zeros(T, 1, dtype=torch.int32, device=DEV), 0, 1, ws)
    M.moe_gather(x, ws, 1, T)
    M.grouped_gemm_gated(ws.xs, wgu, ws.act, ws, T, max_chunks=chunks)
    assert ops.read_status() == 0
    g, u = (x.float() @ wgu[0, h * I:(h + 1) * I].float().t() for h in range(2))
    got = ws.act[ws.pair_pos.long()].float()
    assert _rel(got, torch.nn.functional.silu(g) * u) < 3 * 2.0 ** -8


@pytest.mark.parametrize("T,E,k,H,I", [(512, 8, 2, 256, 1792), (700, 8, 2, 256, 1792), (1024, 8, 2, 256, 1792), (1100, 2, 2, 72, 136)])
def test_grouped_gemm_gated_of_128_and_256_rows(T, E, k, H, I):
    """More than 64 rows an expert: 256 rows a CTA where the CTAs are few, 128 and two CTAs an SM otherwise, chunks of less, of
    exactly and of more than that; the bits of the product and the activation as two kernels."""
    torch.manual_seed(T)
    x = torch.randn(T, H, device=DEV).to(torch.bfloat16)
    wgu = (torch.randn(E, 2 * I, H, device=DEV) * H ** -0.5).to(torch.bfloat16)
    ids = torch.stack([torch.randperm(E, device=DEV)[:k] for _ in range(T)]).int()
    ids[:128, 0], ids[:128, 1:] = 0, 1                    # an expert that shares rows with few others
    ws = M.MoeWorkspace(torch.device(DEV), T, k, E, H, I)
    M.moe_sort(ids, 0, E, ws)
    P = T * k
    M.moe_gather(x, ws, E, P)
    M.grouped_gemm(ws.xs, wgu, ws.gu, ws, P)
    ops.act_and_mul(ws.gu[:P], 0, out=ws.act[:P])
    want = ws.act[:P].clone()
    ws.act.zero_()
    M.grouped_gemm_gated(ws.xs, wgu, ws.act, ws, P, kind=0)
    assert ops.read_status() == 0 and torch.equal(ws.act[:P], want)
    g, u = (torch.stack([x.float() @ wgu[e, h * I:(h + 1) * I].float().t() for e in range(E)]) for h in range(2))
    tok = torch.arange(T, device=DEV)
    for j in range(k):
        e = ids[:, j].long()
        got = want[ws.pair_pos.view(T, k)[:, j].long()].float()
        assert _rel(got, torch.nn.functional.silu(g[e, tok]) * u[e, tok]) < 3 * 2.0 ** -8


@pytest.mark.parametrize("T,E,I,N", [(300, 2, 1000, 136), (700, 8, 1000, 1024), (1400, 8, 1000, 2048)])
def test_grouped_gemm_of_few_and_of_many_ctas(T, E, I, N):
    """Plain products of more than 64 rows an expert with K longer than the ring: grids of fewer CTAs than SMs (four stages) and of
    more (two stages, two CTAs an SM). fp32 sums, one rounding to bf16."""
    torch.manual_seed(T)
    ws = M.MoeWorkspace(torch.device(DEV), T, 2, E, N, I)
    ids = torch.stack([torch.randperm(E, device=DEV)[:2] for _ in range(T)]).int()
    M.moe_sort(ids, 0, E, ws)
    P = 2 * T
    x = torch.randn(T, I, device=DEV).to(torch.bfloat16)
    wd = (torch.randn(E, N, I, device=DEV) * I ** -0.5).to(torch.bfloat16)
    pos = ws.pair_pos.view(T, 2).long()
    for j in range(2):
        ws.act[pos[:, j]] = x
    M.grouped_gemm(ws.act, wd, ws.y, ws, P)
    assert ops.read_status() == 0
    tok = torch.arange(T, device=DEV)
    y = torch.stack([x.double() @ wd[e].double().t() for e in range(E)])
    for j in range(2):
        assert _rel(ws.y[pos[:, j]].float(), y[ids[:, j].long(), tok].float()) < 2.0 ** -8
    assert bool((ws.y[P:] == 0).all())


@pytest.mark.parametrize("T", [2047, 2048, 3000])
def test_gather_of_few_and_of_many_rows(T):
    """With and without an early start (4096 rows): every sorted row is its token's, rows beyond the sorted ones are untouched."""
    torch.manual_seed(T)
    ws = M.MoeWorkspace(torch.device(DEV), T, 2, 8, 72, 8)
    ids = torch.stack([torch.randperm(8, device=DEV)[:2] for _ in range(T)]).int()
    x = torch.randn(T, 72, device=DEV).to(torch.bfloat16)
    M.moe_sort(ids, 0, 8, ws)
    M.moe_gather(x, ws, 8, 2 * T)
    pos = ws.pair_pos.view(T, 2).long()
    assert torch.equal(ws.xs[pos[:, 0]], x) and torch.equal(ws.xs[pos[:, 1]], x) and bool((ws.xs[2 * T:] == 0).all())


@pytest.mark.parametrize("T,E,H,I,skew", [(700, 8, 72, 136, False), (645, 8, 200, 1000, True), (2600, 4, 64, 128, True),
                                          (4500, 2, 128, 264, False), (257, 2, 2048, 768, False)])
def test_grouped_gemm_of_many_rows_an_expert(T, E, H, I, skew):
    """CTA pairs: ragged weight tiles and k-blocks, chunks of 1 to 256 rows, experts without rows and with more chunks than a group
    (``skew``: every token's second expert is the last one). Each of the two products rounds its values to bf16 (2^-8), the
    gated one three times."""
    torch.manual_seed(T + I)
    x = torch.randn(T, H, device=DEV).to(torch.bfloat16)
    wgu = (torch.randn(E, 2 * I, H, device=DEV) * H ** -0.5).to(torch.bfloat16)
    wd = (torch.randn(E, H, I, device=DEV) * I ** -0.5).to(torch.bfloat16)
    first = torch.randint(0, E - 1, (T,), device=DEV)
    ids = torch.stack([first, torch.full_like(first, E - 1) if skew else (first + 1) % E], 1).int()
    if skew:
        ids[:, 0][ids[:, 0] == 1] = 0                           # (an expert without rows)
    ws = M.MoeWorkspace(torch.device(DEV), T, 2, E, H, I)
    M.moe_sort(ids, 0, E, ws)
    P = 2 * T
    assert P >= 160 * E
    M.moe_gather(x, ws, E, P)
    ws.act.fill_(7.0)
    ws.y.fill_(7.0)
    M.grouped_gemm_gated(ws.xs, wgu, ws.act, ws, P, kind=0)
    M.grouped_gemm(ws.act, wd, ws.y, ws, P)
    assert bool((ws.act[P:] == 7.0).all()) and bool((ws.y[P:] == 7.0).all())        # nothing beyond the sorted rows
    pos = ws.pair_pos.view(T, 2).long()
    for e in range(E):
        at, j = (ids == e).nonzero(as_tuple=True)
        if not at.numel():
            continue
        g, u = (x[at].float() @ wgu[e, h * I:(h + 1) * I].float().t() for h in range(2))
        act, got = torch.nn.functional.silu(g) * u, ws.act[pos[at, j]].float()
        assert ((got - act).norm() / act.norm()).item() < 3 * 2.0 ** -8
        y = got @ wd[e].float().t()
        assert ((ws.y[pos[at, j]].float() - y).norm() / y.norm()).item() < 2.0 ** -8
    assert ops.read_status() == 0


def test_native_attention_half_same_logits_as_per_op_path():
    """The attention halves through the native entry (prefill chunks, mixed steps, decodes): the bits of the per-op path."""
    from vllm_cpp_b200.config import EngineArgs, synthetic_config
    from vllm_cpp_b200.engine import LLM, SamplingParams
    cfg = synthetic_config("tiny-moe")
    cfg.head_dim = 128
    llm = LLM(EngineArgs(model_config=cfg, device="cuda", block_size=16, num_blocks=200, max_model_len=640, max_num_seqs=4,
                         max_num_batched_tokens=160, enable_cuda_graphs=False))
    m, seen = llm.runner.model, []
    assert m._native_attn_ok()
    orig = type(m).forward

    def both(self, ctx):
        self.native_layers = False
        a = orig(self, ctx).clone()
        self.native_layers = True
        seen.append((ctx.num_decodes, ctx.num_prefills, torch.equal(a, orig(self, ctx))))
        return a

    g = torch.Generator().manual_seed(3)
    type(m).forward = both
    try:
        llm.generate([torch.randint(0, cfg.vocab_size, (n,), generator=g).tolist() for n in (200, 9, 70, 150)],
                     SamplingParams(temperature=0.0, max_tokens=5, ignore_eos=True))
    finally:
        type(m).forward = orig
    assert any(nd and npf for nd, npf, _ in seen) and any(nd and not npf for nd, npf, _ in seen)
    assert all(eq for *_, eq in seen), seen
    assert ops.read_status() == 0
