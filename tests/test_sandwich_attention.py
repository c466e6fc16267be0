"""The sandwich arrangement around plain attention on the GPU: results against a float64 statement, and no more kernel
launches in a decode step than if the attention added its result into a zeroed buffer."""
import os

import numpy as np
import pytest
import torch

from plain_llama import plain_attention, plain_inv_freq, plain_rmsnorm, plain_rope, plain_swiglu
from tiny import jitter_norm_weights

pytestmark = pytest.mark.gpu

E, H, K, D, F, V = 256, 32, 8, 64, 128, 97          # the last product of attention sums 2,048 numbers: split over K for a few tokens


def register(block):
    from mdma_b200.config import Architecture
    from mdma_b200.registry import ARCHITECTURES
    from mdma_b200.spec import LayerSpec, ModelSpec, PartSpec, ScheduleEntry

    def describe(c):
        norm = lambda prefix: PartSpec("rmsnorm", dict(width=E, eps=c["eps"]), prefix=prefix)  # noqa: E731
        pos = PartSpec("rotary", dict(head_dim=D, rotary_dim=D, theta=c["theta"], layout="interleaved", scaling=None))
        layers = [LayerSpec(block, norm(f"l{i}.n1."),
                            PartSpec("attention", dict(hidden_size=E, num_heads=H, num_kv_heads=K, head_dim=D, scale=D ** -0.5,
                                                       window=0, position=pos), prefix=f"l{i}.attn."),
                            norm(f"l{i}.n2."), PartSpec("gated_mlp", dict(hidden_size=E, intermediate_size=F), prefix=f"l{i}.mlp."),
                            extras={"mixer_post_norm": norm(f"l{i}.n3."), "ffn_post_norm": norm(f"l{i}.n4.")}) for i in range(2)]
        return ModelSpec(hidden_size=E, vocab_size=V, max_positions=256, embedding=PartSpec("embedding", dict(vocab_size=V, width=E), prefix="emb."),
                         layers=layers, schedule=[ScheduleEntry(0), ScheduleEntry(1)], final_norm=norm("final."),
                         lm_head=PartSpec("lm_head", dict(vocab_size=V, width=E), prefix="head."))

    ARCHITECTURES.register("PlainSandwichLM", Architecture("PlainSandwichLM", lambda d: dict(d), describe), replace=True)


def register_adding():
    """The arrangement without stored results."""
    from mdma_b200.parts.block import SandwichBlock
    from mdma_b200.registry import BLOCKS

    class AddingBlock(SandwichBlock):
        @staticmethod
        def _sublayer(ctx, part, norm, h, x, y, *more):
            y[:ctx.n_tokens].zero_()
            part.forward(ctx, h, y, *more)
            norm.add_normed(ctx, y, x)

    BLOCKS.register("adding_sandwich", AddingBlock, replace=True)


def plain(c, W, ids):
    W = {k: v.double() for k, v in W.items()}
    T = len(ids)
    x = W["emb.weight"][torch.tensor(ids)]
    inv, pos = plain_inv_freq(D, c["theta"], None), torch.arange(T)
    n = lambda v, name: plain_rmsnorm(v, W[name], c["eps"])  # noqa: E731
    for i in range(2):
        p = f"l{i}."
        h = n(x, p + "n1.weight")
        q = plain_rope((h @ W[p + "attn.q_proj.weight"].t()).reshape(T, H, D), pos, inv, "interleaved")
        k = plain_rope((h @ W[p + "attn.k_proj.weight"].t()).reshape(T, K, D), pos, inv, "interleaved")
        v = (h @ W[p + "attn.v_proj.weight"].t()).reshape(T, K, D)
        x = x + n(plain_attention(q, k, v, D ** -0.5) @ W[p + "attn.o_proj.weight"].t(), p + "n3.weight")
        h = n(x, p + "n2.weight")
        x = x + n(plain_swiglu(h @ W[p + "mlp.gate_proj.weight"].t(), h @ W[p + "mlp.up_proj.weight"].t()) @ W[p + "mlp.down_proj.weight"].t(),
                  p + "n4.weight")
    return n(x, "final.weight") @ W["head.weight"].t()


# (bounds of the arrangement's other tests, tests/test_toy_mixer.py: float32 sums; bfloat16 operands of two layers)
@pytest.mark.parametrize("dtype,tol", [("float32", 5e-5), ("bfloat16", 8e-2)])
def test_plain_attention_stores_its_result_between_two_norms(tmp_path, dtype, tol):
    from mdma_b200 import ops
    from mdma_b200.engine import Engine, StepEntry
    from mdma_b200.weights import write_random_model
    from mdma_b200.weights.safetensors_io import SafetensorsFile
    register("sandwich")
    cfg = dict(architectures=["PlainSandwichLM"], eps=1e-5, theta=10000.0)
    d = write_random_model(str(tmp_path / "m"), cfg, 3, torch.bfloat16 if dtype == "bfloat16" else torch.float32, std=0.05)
    jitter_norm_weights(d, 3)
    sf = SafetensorsFile(os.path.join(d, "model.safetensors"))
    W = {n: sf.tensor(n).clone().float() for n in sf.entries}
    g = torch.Generator().manual_seed(2)
    seqs = [torch.randint(0, V, (n,), generator=g).tolist() for n in (70, 9)]
    cut = [50, 3]
    ref = [plain(cfg, W, s).numpy() for s in seqs]
    launches = {}
    register_adding()
    for block in ("sandwich", "adding_sandwich"):
        register(block)
        eng = Engine(d, dtype=dtype, max_batch=2, max_context=128, logit_rows=128)
        slots = [eng.acquire() for _ in seqs]
        out = eng.step([StepEntry(sl, s[:c], list(range(c))) for sl, s, c in zip(slots, seqs, cut)]).cpu().numpy()
        off = 0
        for r, c in zip(ref, cut):
            assert np.abs(out[off:off + c] - r[:c]).max() < tol
            off += c
        for step in range(4):
            before = ops.LAUNCHES
            out = eng.step([StepEntry(sl, [s[c + step]], [0]) for sl, s, c in zip(slots, seqs, cut)]).cpu().numpy()
            launches[block] = ops.LAUNCHES - before
            for row, (r, c) in enumerate(zip(ref, cut)):
                assert np.abs(out[row] - r[c + step]).max() < tol
        eng.check_status()
    assert launches["sandwich"] <= launches["adding_sandwich"]
