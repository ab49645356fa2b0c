"""Edges of the tensor-core GEMMs' work split: rows per tile around the small activation boxes (16, 32) and the full tile,
tiles that several CTAs share along K (linear layer, scaled product, down GEMM), the shared expert's pass, and the kernels
in front of them (fused router + selection, the cluster permutation)."""
import pytest
import torch

from oracle import moe_oracle as O
from tests.gpu_util import small_problem, to_dev

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def m():
    import torch_tpu_b200
    return torch_tpu_b200


def _close(out, want, what):
    """FP8 experts: one e4m3 step of a hidden value (1/16) now and then, as in the other parity tests."""
    met = O.parity_metrics(out, want)
    assert met["max_rel"] <= 2e-2 and met["cosine"] >= 0.9995, (what, met)


@pytest.mark.parametrize("rows", [(1, 15, 16, 17), (31, 32, 33, 0), (112, 113, 127, 128), (129, 145, 161, 5)])
def test_rows_per_tile(m, rows):
    H, I, E = 512, 256, 4
    T = sum(rows)
    p = small_problem(T, H, I, E, 1, seed=T)
    p["ids"] = torch.repeat_interleave(torch.arange(E), torch.tensor(rows)).to(torch.int32)[torch.randperm(T)].view(T, 1).contiguous()
    d = to_dev(p)
    want = O.experts_w8a8(p["x"], p["ids"], p["wg"], p["wu"], p["wd"], p["sg"], p["su"], p["sd"])
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    out = torch.full((T, 1, H), float("nan"), dtype=torch.bfloat16, device=DEV)
    m.ops.experts(out, d["x"], d["wg"], d["wu"], d["wd"], d["sg"], d["su"], d["sd"], d["ids"], status=status)
    assert int(status.item()) == 0
    _close(out, want, rows)


@pytest.mark.parametrize("M,K,N", [(1, 4096, 512), (7, 4096, 1024), (33, 8192, 256), (130, 8192, 576), (300, 16384, 512)])
def test_linear_with_shared_tiles(m, M, K, N):
    """Few tiles with long K loops: every tile is cut along K.  Against an fp64 product of what the kernel multiplies;
    the tolerance is the bf16 rounding of the result (2^-8 of the row's scale) plus the tensor core's 128-deep sums.
    Run twice: the order of the parts does not depend on which CTA comes last."""
    g = torch.Generator().manual_seed(M + K + N)
    x = torch.randn(M, K, generator=g).to(torch.bfloat16)
    w, s = m.weights.quantize_blockwise(torch.randn(N, K, generator=g) * 0.02)
    out = m.ops.linear_w8(x.to(DEV), w.to(DEV), s.to(DEV))
    again = m.ops.linear_w8(x.to(DEV), w.to(DEV), s.to(DEV))
    assert torch.equal(out, again)
    q, st = m.ops.quant_rows(x.to(DEV))
    xs = (q.double().view(M, K // 128, 128) * st[:, :M].t().double().unsqueeze(-1)).view(M, K)
    wf = w.to(DEV).double() * s.to(DEV).double().repeat_interleave(128, 0)[:N].repeat_interleave(128, 1)
    want = xs @ wf.t()
    err = (out.double() - want).abs().max() / want.pow(2).mean().sqrt()
    assert float(err) <= 4 * 2.0 ** -8 + 5e-3, float(err)


def test_few_tokens_with_a_long_gate_up_k_loop_are_reproducible(m):
    """Six tokens, 32 K blocks in the gate/up GEMM and two in the down GEMM (neither cuts a tile or splits K): calls give
    equal bits.  Cut tiles: test_down_gemm_with_shared_tiles_and_a_capped_grid, test_linear_with_shared_tiles."""
    H, I, E, T = 4096, 256, 4, 6
    p = small_problem(T, H, I, E, 2, seed=8)
    d = to_dev(p)
    outs = []
    for _ in range(3):
        out = torch.full((T, 2, H), float("nan"), dtype=torch.bfloat16, device=DEV)
        m.ops.experts(out, d["x"], d["wg"], d["wu"], d["wd"], d["sg"], d["su"], d["sd"], d["ids"])
        outs.append(out)
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    _close(outs[0], O.experts_w8a8(p["x"], p["ids"], p["wg"], p["wu"], p["wd"], p["sg"], p["su"], p["sd"]), "gate/up")


def _ragged(E, T, k, seed):
    """ids of T tokens over E experts with very uneven loads (experts without rows, one with more than one m-tile)."""
    g = torch.Generator().manual_seed(seed)
    p = torch.rand(E, generator=g) ** 4
    p[0], p[1] = p.sum(), 0.0
    return torch.stack([torch.multinomial(p, k, generator=g) for _ in range(T)]).to(torch.int32)


@pytest.mark.parametrize("cap", [1, 7, 98, 147])
def test_down_gemm_with_shared_tiles_and_a_capped_grid(m, cap):
    """E <= 40 tiles of 12 K blocks on 148 SMs: the down GEMM cuts each along K.  Which tiles are cut does not depend on
    max_ctas (a CTA then walks several parts), so every cap gives the bits of the whole grid, and a second call too."""
    T, H, I, E, k = 300, 256, 1536, 40, 2
    p = small_problem(T, H, I, E, k, seed=21)
    p["ids"] = _ragged(E, T, k, 4)
    d = to_dev(p)
    outs = []
    for c in (0, cap, cap):
        out = torch.full((T, k, H), float("nan"), dtype=torch.bfloat16, device=DEV)
        status = torch.zeros(1, dtype=torch.int32, device=DEV)
        m.ops.experts(out, d["x"], d["wg"], d["wu"], d["wd"], d["sg"], d["su"], d["sd"], d["ids"], status=status,
                      max_ctas=c)
        assert int(status.item()) == 0
        outs.append(out)
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    _close(outs[0], O.experts_w8a8(p["x"], p["ids"], p["wg"], p["wu"], p["wd"], p["sg"], p["su"], p["sd"]), cap)


@pytest.mark.parametrize("M,K,N", [(1, 4096, 512), (40, 2048, 1088), (130, 8192, 576)])
def test_scaled_mm_fp32_rows_with_shared_tiles(m, M, K, N):
    """fp32 result rows of tiles that are cut along K.  Every product of two e4m3 values is exact; tolerance as in the
    uncut test: fp32 sums, 1e-5 of the largest result."""
    m.load_ops()
    g = torch.Generator().manual_seed(M)
    x = (torch.rand(M, K, generator=g) * 2 - 1).to(torch.float8_e4m3fn)
    y = (torch.rand(K, N, generator=g) * 2 - 1).to(torch.float8_e4m3fn)
    outs = [torch.ops.my_ops._scaled_mm(x.to(DEV), y.t().contiguous().to(DEV), torch.tensor(0.5), torch.tensor(3.0), None,
                                        None, torch.float32, False) for _ in range(2)]
    assert torch.equal(*outs)
    met = O.parity_metrics(outs[0].cpu(), x.double() @ y.double() * 1.5)
    assert met["max_rel"] <= 1e-5 and met["cosine"] >= 0.99999, met


@pytest.mark.parametrize("T,E,k", [(1, 4, 2), (9, 8, 2), (130, 3, 2), (700, 8, 3)])
@pytest.mark.parametrize("I_shared", [256, 384])
@pytest.mark.parametrize("fused", [False, True])
def test_shared_expert_beside_and_in_line(m, T, E, k, I_shared, fused):
    """The shared expert, of the routed experts' size and of another: beside them on a side stream (up to 64 tokens) or
    behind them.  Also with an id out of range, whose dropped row must not move the shared expert's."""
    H, I = 512, 256
    p = small_problem(T, H, I, E, k, seed=T + E)
    sh = O.make_expert_weights(1, H, I_shared, seed=99)
    if T > 1:
        p["ids"][1, 0] = E
    d = to_dev(p)
    out = torch.full((T, H), float("nan"), dtype=torch.bfloat16, device=DEV)
    m.ops.experts(out, d["x"], d["wg"], d["wu"], d["wd"], d["sg"], d["su"], d["sd"], d["ids"], d["w"],
                  shared=tuple(t.to(DEV) for t in sh), fused_combine=fused)
    w = p["w"].clone()
    ids = p["ids"].clone()
    if T > 1:
        w[1, 0], ids[1, 0] = 0.0, 0
    y = O.experts_w8a8(p["x"], ids, p["wg"], p["wu"], p["wd"], p["sg"], p["su"], p["sd"]).float()
    s = O.experts_w8a8(p["x"], torch.zeros(T, 1, dtype=torch.int32), *sh).float()
    _close(out, (y * w[..., None]).sum(1) + s[:, 0], (T, E, k, I_shared, fused))


@pytest.mark.parametrize("T", [1, 4, 5, 33])
@pytest.mark.parametrize("E,k", [(2, 1), (8, 2), (9, 3), (16, 16), (17, 4)])
def test_router_route_is_the_two_calls(m, T, E, k):
    H = 520
    x, wr, _ = O.make_inputs(T, H, E, seed=T + E, router_std=H ** -0.5)
    x, wr = x.to(DEV), wr.to(DEV)
    bias = torch.randn(E, generator=torch.Generator().manual_seed(1)).to(DEV) * 0.1
    for score, b, lb in (("softmax", None, bias), ("sigmoid", bias, None)):
        logits = torch.full((T, E), float("nan"), device=DEV)
        ids, w = m.ops.router_route(x, wr, k, score, b, 1, 1, True, 2.5, logits=logits, logit_bias=lb)
        want = m.ops.route(logits, k, score, b, 1, 1, True, 2.5, logit_bias=lb)
        assert torch.equal(ids, want[0]) and torch.equal(w, want[1])
        ref = x.double() @ wr.double().T
        assert float((logits.double() - ref).abs().max()) <= 2e-6 * float(ref.abs().max())


@pytest.mark.parametrize("T", [17, 64, 591, 592, 593, 600])
@pytest.mark.parametrize("E,k,groups,topk_groups", [(8, 2, 1, 1), (16, 4, 4, 2), (64, 6, 8, 3)])
def test_router_route_with_groups_and_around_one_block_per_sm(m, T, E, k, groups, topk_groups):
    """Up to 4 tokens per SM (592) and 16 experts one kernel routes too, above that a second one: the same logits, ids and
    weights as the two calls, with groups as well."""
    H = 256
    x, wr, _ = O.make_inputs(T, H, E, seed=T + E, router_std=H ** -0.5)
    x, wr = x.to(DEV), wr.to(DEV)
    bias = torch.randn(E, generator=torch.Generator().manual_seed(2)).to(DEV) * 0.1
    for score, b in (("softmax", None), ("sigmoid", bias)):
        logits = torch.full((T, E), float("nan"), device=DEV)
        ids, w = m.ops.router_route(x, wr, k, score, b, groups, topk_groups, True, 1.5, logits=logits)
        assert torch.equal(logits, m.ops.router_logits(x, wr))
        want = m.ops.route(logits, k, score, b, groups, topk_groups, True, 1.5)
        assert torch.equal(ids, want[0]) and torch.equal(w, want[1])


@pytest.mark.parametrize("P,E", [(1024, 8), (1025, 8), (2048, 1000), (8191, 128), (8192, 1024), (8193, 64)])
def test_permutation_around_its_kernel_sizes(m, P, E):
    g = torch.Generator().manual_seed(P + E)
    ids = torch.randint(-1, E + 1, (P, 1), generator=g, dtype=torch.int32)  # some out of range
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    order, offs = m.ops.permute(ids.to(DEV), E, status=status)
    flat = ids.view(-1).long()
    ok = (flat >= 0) & (flat < E)
    want = torch.argsort(torch.where(ok, flat, torch.full_like(flat, E)), stable=True)
    n = int(ok.sum())
    assert torch.equal(order.cpu()[:n].long(), want[:n]) and bool((order[n:] == -1).all())
    assert torch.equal(offs.cpu().long(), torch.cat([torch.zeros(1, dtype=torch.long), torch.bincount(flat[ok], minlength=E).cumsum(0)]))
    assert int(status.item()) == (1 if n < P else 0)
