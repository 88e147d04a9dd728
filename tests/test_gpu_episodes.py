"""Episodes stacked along the rows: each keeps the bits of a stack of its own; the split-K planes for
more than 128 rows are those of the skinny form."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
E4M3 = torch.float8_e4m3fn


# a second row block of one row, a ragged last column tile, K not a whole number of stages per range, a
# narrow output (64-wide tiles), one range
@pytest.mark.parametrize("M,N,K,S", [(129, 1024, 4096, 8), (400, 1040, 2688, 5), (300, 272, 1664, 3), (200, 208, 512, 1), (1030, 768, 1024, 2)])
def test_planes_do_not_depend_on_the_rows(M, N, K, S):
    from instinctflash_b200.kernels import fp8
    g = torch.Generator(device=DEV).manual_seed(M)
    a = torch.randn(M, K, device=DEV, generator=g).to(E4M3)
    w = fp8.Fp8Weight(torch.randn(N, K, device=DEV, generator=g).to(E4M3), torch.ones(N, device=DEV), None)
    planes = torch.full((S, M, N), float("nan"), device=DEV)
    fp8.gemm_partials(a, w, planes)
    for lo in (0, max(0, M - 128)):
        rows = a[lo:lo + 128]
        want = torch.empty(S, rows.shape[0], N, device=DEV)
        fp8.gemm_partials(rows, w, want)
        torch.cuda.synchronize()
        assert torch.equal(planes[:, lo:lo + 128], want)
    assert not torch.isnan(planes).any()
    exact = a.double() @ w.w.double().T   # fp32 accumulation of K exact products
    assert ((planes.double().sum(0) - exact).norm() / exact.norm()).item() < 1e-5


@pytest.mark.parametrize("M,hidden,ffn,o_in,episodes", [(33, 768, 2688, 2048, 3), (128, 1024, 2560, 0, 2), (8, 1280, 5120, 2048, 5)])
def test_episode_batch_bits(M, hidden, ffn, o_in, episodes):
    from instinctflash_b200.stack import EpisodeBatch, LinearStack, StackSpec, make_inputs, make_weights
    spec = StackSpec("expert", "gemma", 2, M, hidden, ffn, 1536, o_in=o_in, seed=6)
    weights = make_weights(spec, DEV)
    xs = [make_inputs(StackSpec(**{**spec.__dict__, "seed": 60 + e}), DEV)[0] for e in range(episodes)]
    attn = make_inputs(spec, DEV)[1]
    want = []
    for x in xs:
        st = LinearStack(spec, weights, DEV)
        st.load(x, attn)
        want.append(st.forward().clone())
    batch = EpisodeBatch(spec, weights, DEV, episodes)
    batch.load(xs, attn)
    g = batch.capture()
    batch.load(xs, attn)
    g.replay()
    torch.cuda.synchronize()
    for st, w in zip(batch.stacks, want):
        assert torch.equal(st.res, w)
    for st, x, w in zip(batch.stacks, xs, want):   # an episode by itself, on its rows of the batch's buffers
        st.load(x, attn)
        assert torch.equal(st.forward(), w)
