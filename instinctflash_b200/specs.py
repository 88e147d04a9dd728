"""Shapes of the layer stacks: what ``stack.py`` runs and the benchmark names.  No kernels here, so that a
program which needs only the shapes loads none."""
from __future__ import annotations

from dataclasses import dataclass


@dataclass(frozen=True)
class StackSpec:
    name: str
    kind: str            # "gemma" | "wan"
    layers: int
    M: int
    hidden: int
    ffn: int
    qkv: int
    o_in: int = 0        # width of the attention output fed to the O projection (0: no O projection)
    cross: bool = False  # wan: cross-attention q / o projections
    steps: int = 1       # flow steps (the expert re-reads every weight each step)
    sigma: float = 0.02
    outlier_frac: float = 0.0
    outlier_scale: float = 1.0
    seed: int = 0

    def linears(self):
        """(name, N, K) of the FP8 GEMMs of one layer, in call order."""
        out = [("qkv", self.qkv, self.hidden)]
        if self.o_in:
            out.append(("o", self.hidden, self.o_in))
        if self.cross:
            out += [("cross_q", self.hidden, self.hidden), ("cross_o", self.hidden, self.hidden)]
        if self.kind == "gemma":
            out += [("gate_up", 2 * self.ffn, self.hidden), ("down", self.hidden, self.ffn)]
        else:
            out += [("ff1", self.ffn, self.hidden), ("ff2", self.hidden, self.ffn)]
        return out

    def flops(self) -> float:
        return 2.0 * self.M * sum(n * k for _, n, k in self.linears()) * self.layers * self.steps

    def weight_bytes(self) -> float:
        return float(sum(n * k for _, n, k in self.linears()) * self.layers)


SPECS = {
    # pi05 PaliGemma prefix (Gemma-2B): 18 layers, M = 3*256 image + 48 text tokens
    "c2": StackSpec("c2", "gemma", 18, 816, 2048, 16384, 2560, o_in=2048, outlier_frac=0.01, outlier_scale=20.0, seed=1),
    # pi05 action expert (Gemma-300M shape), 10 flow steps, M = 50 action tokens per episode
    "c3": StackSpec("c3", "gemma", 18, 50, 1024, 4096, 1536, steps=10, seed=2),
    # the reference engine's true expert shapes (fused QKV 2560, O projection 2048 -> 1024)
    "c3ref": StackSpec("c3ref", "gemma", 18, 50, 1024, 4096, 2560, o_in=2048, steps=10, seed=2),
    # LingBot-VA / Wan2.2-5B-shape DiT
    "c4": StackSpec("c4", "wan", 30, 4680, 3072, 14336, 9216, o_in=3072, cross=True, outlier_frac=0.005,
                    outlier_scale=30.0, seed=3),
    # DreamZero / Wan-14B-shape DiT, CFG batch 2 x 8192 tokens
    "c5": StackSpec("c5", "wan", 40, 16384, 5120, 13824, 15360, o_in=5120, sigma=0.015, outlier_frac=0.005,
                    outlier_scale=30.0, seed=4),
}


def small_spec(spec: StackSpec, layers: int = 2, M: int | None = None) -> StackSpec:
    """Same layer geometry, fewer layers / rows: the parity-test size."""
    return StackSpec(**{**spec.__dict__, "layers": layers, "M": M if M is not None else spec.M,
                        "name": spec.name + "_small"})
