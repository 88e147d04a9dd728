"""The two-kernel dynamic pack on either side of the size that its grid holds in one pass, with ragged ends and off the
16-byte rule: the recipe's own division."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
E4M3 = torch.float8_e4m3fn


@pytest.mark.parametrize("n", [1, 7, 8193, 524297, 8388600, 8388608, 8388609, 8388616, 9000001])
@pytest.mark.parametrize("shift", [0, 1])
def test_one_pass_and_more(n, shift):
    from instinctflash_b200 import _lib
    g = torch.Generator(device=DEV).manual_seed(n)
    x = torch.randn(n + shift, device=DEV, generator=g).to(torch.bfloat16)[shift:]
    x[n - 1] = 30.0   # the maximum is the last element
    q, s = torch.full((n + 8,), 0x55, device=DEV, dtype=torch.uint8), torch.empty(1, device=DEV)
    for scale in (1.0, 1e-3):   # behind a kernel that has just written x
        x.mul_(scale)
        assert _lib.lib().iflb200_dynamic_pack_bf16_e4m3_noalloc(x.data_ptr(), n, q.data_ptr(), s.data_ptr(),
                                                                torch.cuda.current_stream().cuda_stream) == 0
        want_s = x.float().abs().amax().clamp_min(1e-12).reshape(1) / 448.0
        want = (x.float() / want_s).clamp(-448, 448).to(E4M3).view(torch.uint8)
        assert torch.equal(s.view(torch.int32), want_s.view(torch.int32)) and torch.equal(q[:n], want) and (q[n:] == 0x55).all()


@pytest.mark.parametrize("n_rows", [1024, 3000])   # of 1024: 2^20 elements and just under three times as many
def test_packs_one_behind_the_other_on_one_buffer(n_rows):
    """Producer, maxima, pack, producer, maxima, pack without a pause, eagerly and captured: a pack reads its elements ahead of its
    own wait, and must read what the producer directly before has written, not what the buffer held."""
    from instinctflash_b200.kernels import fp8
    from instinctflash_b200.runtime.fp8_pack import dynamic_pack_bf16_e4m3
    g = torch.Generator(device=DEV).manual_seed(n_rows)
    w = fp8.Fp8Weight(torch.randn(1024, 512, device=DEV, generator=g).to(E4M3), None, None)
    acts = [(torch.randn(n_rows, 512, device=DEV, generator=g) * (1 + i)).to(E4M3) for i in range(4)]
    x = torch.zeros(n_rows, 1024, device=DEV, dtype=torch.bfloat16)

    def chain(sync=lambda: None):
        outs = []
        for a in acts:
            fp8.gemm(a, w, x)
            sync()
            outs += dynamic_pack_bf16_e4m3(x)
            sync()
        return outs

    want = [t.clone() for t in chain(torch.cuda.synchronize)]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = chain()
    for launch in (chain, lambda: graph.replay() or captured, chain, lambda: graph.replay() or captured):
        x.zero_()
        outs = launch()
        torch.cuda.synchronize()
        assert all(torch.equal(a.view(torch.uint8), b.view(torch.uint8)) for a, b in zip(outs, want))
