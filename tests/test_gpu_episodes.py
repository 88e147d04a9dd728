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


@pytest.mark.parametrize("M,o_in", [(50, 0), (150, 2048)])
def test_episodes_on_streams_of_their_own(M, o_in):
    """All loaded first, then each by itself beside the others: planes, codes and accumulators of one are not
    another's to write."""
    from instinctflash_b200.stack import EpisodeBatch, LinearStack, StackSpec, make_inputs, make_weights
    spec = StackSpec("expert", "gemma", 3, M, 1024, 4096, 1536, o_in=o_in, seed=6)
    weights = make_weights(spec, DEV)
    xs = [make_inputs(StackSpec(**{**spec.__dict__, "seed": 70 + e}), DEV)[0] for e in range(3)]
    attn = make_inputs(spec, DEV)[1]
    batch = EpisodeBatch(spec, weights, DEV, 3)
    want = []
    for x in xs:   # K cut as the batch cuts it
        st = LinearStack(spec, weights, DEV, split_rows=M if M <= 128 else 3 * M)
        st.load(x, attn)
        want.append(st.forward().clone())
    for _ in range(3):
        batch.load(xs, attn)
        streams = [torch.cuda.Stream() for _ in xs]
        torch.cuda.synchronize()
        for st, s in zip(batch.stacks, streams):
            with torch.cuda.stream(s):
                st.forward()
        torch.cuda.synchronize()
        for st, w in zip(batch.stacks, want):
            assert torch.equal(st.res, w)


# one column block wider than the residual kernel over planes takes, and the widest that it takes
@pytest.mark.parametrize("hidden", [9216, 8192])
def test_wide_decoder_stack_above_128_rows(hidden):
    from instinctflash_b200.stack import LinearStack, StackSpec, make_inputs, make_weights
    spec = StackSpec("wide", "gemma", 1, 129, hidden, 16384, 512, seed=8)
    weights = make_weights(spec, DEV)
    x, attn = make_inputs(spec, DEV)
    got = []
    for planes in (True, False):
        st = LinearStack(spec, weights, DEV, split_partials=planes)
        st.load(x, attn)
        got.append(st.forward().double())
    # the order of the K sum may differ, which can move a sum across a bf16 rounding: 2^-8 of the update's size
    update = got[1] - x.double()
    assert ((got[0] - got[1]).norm() / update.norm()).item() < 2.0 ** -8


# the 64-row form and its neighbours, and K whose last slab is ragged: with whole stages in front, alone in its
# stage, in the first stage; the K order does not depend on the form, so the bits are those of 128-wide tiles
@pytest.mark.parametrize("M", [1, 16, 17, 50, 63, 64, 65, 128, 300])
@pytest.mark.parametrize("K", [400, 512, 528, 1040, 1152, 2032])
def test_skinny_forms_bits(M, K):
    from instinctflash_b200 import _lib
    from instinctflash_b200.kernels import fp8
    g = torch.Generator(device=DEV).manual_seed(K)
    N = 336
    a = torch.full((M + 1, K), 448.0, device=DEV).to(E4M3)   # a row behind the operand must not be read into it
    a[:M] = torch.randn(M, K, device=DEV, generator=g).to(E4M3)
    wt = torch.full((N + 1, K), 448.0, device=DEV).to(E4M3)
    wt[:N] = torch.randn(N, K, device=DEV, generator=g).to(E4M3)
    w = fp8.Fp8Weight(wt[:N], torch.rand(N, device=DEV, generator=g), torch.randn(N, device=DEV, generator=g))
    s = torch.rand(M, device=DEV, generator=g)
    outs = []
    for tile in (64, 128):
        assert _lib.lib().iflb200_gemm_set_config(tile, 0, 0) == 0 and _lib.lib().iflb200_gemm_set_split_k(1) == 0
        try:
            raw = torch.full((M, N), float("nan"), device=DEV, dtype=torch.bfloat16)
            fp8.gemm(a[:M], w, raw)
            y = [torch.full((M, N), float("nan"), device=DEV, dtype=t) for t in (torch.float32, torch.float16)]
            for o in y:
                fp8.fp8_linear(a[:M], s, w, o)
            torch.cuda.synchronize()
            outs.append([raw, *y])
        finally:
            _lib.lib().iflb200_gemm_set_config(0, 0, 0)
            _lib.lib().iflb200_gemm_set_split_k(0)
    for p, q in zip(*outs):
        assert not torch.isnan(p).any() and torch.equal(p, q)
    exact = (a[:M].double() @ wt[:N].double().T)   # exact products: the bf16 rounding of an fp32 sum
    assert ((outs[0][0].double() - exact).abs() <= 2.0 ** -8 * exact.abs() + 1e-4 * K ** 0.5).all()
