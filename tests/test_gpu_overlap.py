"""Kernels of a call overlap the end of their predecessor: what such an early start must not take from others."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def m():
    import torch_tpu_b200
    return torch_tpu_b200


def _raw_weights(E, H, I, seed):
    """Random finite e4m3 bytes (exponent at most 2^0) with small block scales: values are not the point here."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    w = []
    for _ in range(3):
        b = torch.randint(0, 256, (E, I, H), generator=g, device=DEV, dtype=torch.uint8)
        w.append((b & 0xBF).view(torch.float8_e4m3fn))
        del b
    s = [torch.full((E, I // 128, H // 128), 2.0 ** -6, device=DEV) for _ in range(3)]
    return (*w, *s)


@pytest.mark.parametrize("tokens", [2048, 4096])
def test_capped_grid_leaves_sms_to_another_stream(m, tokens):
    """max_ctas = n: the other SMs stay free for another stream's kernels for as long as the call runs.  The gate/up GEMM
    of one expert on 98 SMs takes hundreds of microseconds and is two thirds of the call; a permutation on another
    stream takes tens.  If the down GEMM's CTAs, or the kernels behind them, already sit on the free SMs and wait, the
    permutation cannot end before the gate/up GEMM does."""
    H, I, E = 4096, 14336, 1
    w = _raw_weights(E, H, I, 5)
    x = torch.randn(tokens, H, device=DEV).to(torch.bfloat16)
    ids = torch.zeros(tokens, 1, dtype=torch.int32, device=DEV)
    out = torch.empty(tokens, 1, H, dtype=torch.bfloat16, device=DEV)
    other = torch.randint(0, 64, (1024, 4), dtype=torch.int32, device=DEV)
    d = m.ops.make_desc(tokens, H, I, E, 1, max_ctas=98)
    ws = torch.empty(m.ops.experts_workspace_bytes(d) + 256, dtype=torch.uint8, device=DEV)
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(3)]
    torch.cuda.synchronize()
    shares = []
    for _ in range(5):
        with torch.cuda.stream(a):
            ev[0].record()
            m.ops.experts(out, x, *w, ids, workspace=ws, max_ctas=98)
            ev[1].record()
        with torch.cuda.stream(b):
            m.ops.permute(other, 64)
            ev[2].record()
        torch.cuda.synchronize()
        shares.append(ev[0].elapsed_time(ev[2]) / ev[0].elapsed_time(ev[1]))
    assert sorted(shares)[2] < 0.5, shares


def test_wait_limits_do_not_count_the_predecessors_time(m):
    """The bounded waits of a GEMM give up after about a second.  That second is for its own progress: a gate/up GEMM that
    takes longer (here one CTA walks 4 million K blocks, about two seconds) must not make the down GEMM behind it give
    up, whether or not it was started early."""
    T, H, I, E = 8191, 16384, 65536, 1
    w = _raw_weights(E, H, I, 6)
    x = torch.randn(T, H, device=DEV).to(torch.bfloat16)
    ids = torch.zeros(T, 1, dtype=torch.int32, device=DEV)
    outs = []
    for cap in (0, 1):
        out = torch.full((T, 1, H), float("nan"), dtype=torch.bfloat16, device=DEV)
        status = torch.zeros(1, dtype=torch.int32, device=DEV)
        t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        t0.record()
        m.ops.experts(out, x, *w, ids, status=status, max_ctas=cap)
        t1.record()
        torch.cuda.synchronize()
        assert int(status.item()) == 0, cap
        assert torch.isfinite(out.float()).all(), cap
        outs.append(out)
    assert t0.elapsed_time(t1) > 2000  # (two thirds of it in the gate/up GEMM: beyond the limit, or this shows nothing)
    assert torch.equal(*outs)  # (which tiles are cut along K does not depend on the cap)
