"""Host-side logic of the episode batch on CPU (operators of the CPU oracle): an episode of a stacked batch
behaves like a stack of its own, whatever the other episodes do."""
from types import SimpleNamespace

import pytest
import torch

import oracle_ops
from instinctflash_b200.stack import EpisodeBatch, LinearStack, StackSpec, make_inputs, make_weights

EPISODES = 3


def split_ops(planes=2):
    """The oracle's operators with K-split GEMMs, as this package's operator set has them."""
    ops = oracle_ops.ops()

    def gemm_partials(a, w, out):
        cuts = [a.shape[1] * i // out.shape[0] for i in range(out.shape[0] + 1)]
        for plane, lo, hi in zip(out, cuts, cuts[1:]):
            part = oracle_ops.CpuFp8Weight(w.w[:, lo:hi].contiguous(), None)
            oracle_ops.gemm_acc(a[:, lo:hi].contiguous(), part, plane)

    ops.gemm_partials, ops.partial_splits = gemm_partials, lambda M, N, K, sms: planes
    return ops


@pytest.fixture
def setup(monkeypatch):
    monkeypatch.setattr(torch.cuda, "get_device_properties", lambda dev: SimpleNamespace(multi_processor_count=148))

    def make(o_in):
        spec = StackSpec("tiny", "gemma", layers=2, M=8, hidden=64, ffn=128, qkv=96, o_in=o_in, seed=5)
        weights = make_weights(spec, "cpu", cpu_seeded=True)
        xs = [make_inputs(StackSpec(**{**spec.__dict__, "seed": 50 + e}), "cpu")[0] for e in range(EPISODES)]
        attn = make_inputs(spec, "cpu")[1]
        lone = [LinearStack(spec, weights, "cpu", ops=split_ops()) for _ in range(EPISODES)]
        for st, x in zip(lone, xs):
            st.load(x, attn)
        batch = EpisodeBatch(spec, weights, "cpu", EPISODES, ops=split_ops())
        assert batch.merged is not None
        return batch, lone, xs, attn
    return make


# no output projection: load()'s codes feed the feed-forward; codes of the attention output in the residual
# stream's width, and in one of their own
@pytest.mark.parametrize("o_in", [0, 64, 96])
@pytest.mark.parametrize("whole", [True, False])
def test_episodes_loaded_together_run_one_by_one(setup, o_in, whole):
    batch, lone, xs, attn = setup(o_in)
    if whole:
        batch.load(xs, attn)
    else:
        for st, x in zip(batch.stacks, xs):
            st.load(x, attn)
    for st, alone in zip(batch.stacks, lone):
        assert torch.equal(st.forward(), alone.forward())
    for st, alone in zip(batch.stacks, lone):   # nothing of an episode's result was the others' to write
        assert torch.equal(st.res, alone.res)


def test_episode_and_batch_take_turns(setup):
    batch, lone, xs, attn = setup(0)
    batch.load(xs, attn)
    batch.stacks[1].forward()
    lone[1].forward()
    batch.forward()
    batch.stacks[2].forward()
    lone[2].forward()
    for st, alone in zip(batch.stacks, lone):
        assert torch.equal(st.res, alone.forward())


def test_scratch_of_an_episode_is_its_own(setup):
    batch, _, xs, attn = setup(0)
    batch.load(xs, attn)
    for st in batch.stacks:
        st.forward()
    for name in ("q8", "raw", "part"):
        used = [getattr(st, name) for st in batch.stacks] + [getattr(batch.merged, name)]
        spans = sorted((t.data_ptr(), t.data_ptr() + t.numel() * t.element_size()) for t in used)
        assert all(a[1] <= b[0] for a, b in zip(spans, spans[1:])), name


def test_fewer_inputs_than_episodes(setup):
    """As with separate stacks, the episodes behind the last input keep what they have."""
    batch, lone, xs, attn = setup(64)
    batch.load(xs, attn)
    batch.load(xs[1:2], attn)
    lone[0].load(xs[1], attn)
    batch.load([], attn)
    batch.forward()
    for st, alone in zip(batch.stacks, lone):
        assert torch.equal(st.res, alone.forward())


def test_attention_outputs_of_several_types(setup):
    batch, lone, xs, attn = setup(64)
    batch.load(xs, attn)
    for e, dtype in enumerate((torch.float16, torch.bfloat16, torch.float32)):
        mine = (attn.float() * (1.0 + e / 7)).to(dtype)
        batch.stacks[e].load(xs[e], mine)
        lone[e].load(xs[e], mine)
    batch.forward()
    for st, alone in zip(batch.stacks, lone):
        assert torch.equal(st.res, alone.forward())


def test_attention_buffer_of_a_captured_pass_stays(setup):
    """A captured graph writes to the addresses of its capture: changing the element type in between must not
    free them."""
    batch, _, xs, attn = setup(64)
    used = []
    for dtype in (torch.bfloat16, torch.float16, torch.bfloat16):
        batch.load(xs, attn.to(dtype))
        batch.forward()
        used.append(batch.merged.attn.data_ptr())
    assert used[0] == used[2] != used[1]


@pytest.mark.parametrize("bad", [lambda t: t[:1], lambda t: t.double(), lambda t: t.to("meta"), lambda t: t.T.contiguous().T])
def test_attention_outputs_that_one_stack_refuses(setup, bad):
    batch, _, xs, attn = setup(64)
    batch.load(xs, bad(attn))
    with pytest.raises(ValueError):
        batch.forward()


def test_no_planes_are_held_where_nothing_is_split(monkeypatch):
    monkeypatch.setattr(torch.cuda, "get_device_properties", lambda dev: SimpleNamespace(multi_processor_count=148))
    spec = StackSpec("tiny", "gemma", layers=1, M=8, hidden=64, ffn=128, qkv=96, seed=5)
    weights = make_weights(spec, "cpu", cpu_seeded=True)
    held = [LinearStack(spec, weights, "cpu", ops=split_ops(planes)).part.numel() for planes in (1, 2)]
    assert held == [0, 2 * spec.M * spec.hidden]


def test_launches_of_a_stacked_pass_count_once(setup):
    batch, lone, xs, attn = setup(64)
    batch.load(xs, attn)
    batch.forward()
    lone[0].forward()
    assert batch.launches_per_forward == lone[0].launches_per_forward
