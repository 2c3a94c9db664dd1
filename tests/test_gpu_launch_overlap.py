"""Kernels launched so that they may start while their predecessor ends, over whole steps of small models of every design: the same
bits as launched one after the other, kernel by kernel and in captured steps."""
from __future__ import annotations

import importlib

import pytest
import torch

from gpu_util import DEV

pytestmark = pytest.mark.gpu

# wide enough that a float32 run's products go to the kernels made for them (2^20 weights each)
WIDE = dict(architectures=["Qwen3ForCausalLM"], num_hidden_layers=2, hidden_size=1024, num_attention_heads=8, num_key_value_heads=2,
            head_dim=128, intermediate_size=1536, vocab_size=1100, rope_theta=1e6, rms_norm_eps=1e-6, tie_word_embeddings=False,
            attention_bias=False, max_position_embeddings=4096)


def configs():
    yield "qwen3", WIDE
    for design in ("romepel", "zevivik", "pikalorn", "vodalorn", "gekilix", "vuvalorn"):
        for name, cfg in importlib.import_module(f"test_gpu_{design}").CONFIGS.items():
            yield f"{design}-{name}", cfg


CONFIGS = dict(configs())


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("name", list(CONFIGS))
def test_steps_have_the_same_bits(name, dtype):
    """Prompts of unequal lengths, a short portion of one sequence, two portions beside each other, decode steps of three and
    of one."""
    from nncpu_b200 import Engine, Model
    from nncpu_b200.config import config_from_dict
    from nncpu_b200.engine.model import parameter_list
    from nncpu_b200.kernels import ops
    from nncpu_b200.parts import Runtime
    from nncpu_b200.weights import random_tensors_on_device
    cfg, dt = config_from_dict(dict(CONFIGS[name])), getattr(torch, dtype)
    model = Model(cfg, random_tensors_on_device(parameter_list(cfg.model_spec()), 3, dt, DEV), Runtime(DEV, dt))
    vocab = cfg.model_spec().vocab_size

    def ids(n, seed):
        return torch.randint(0, vocab, (n,), generator=torch.Generator().manual_seed(seed)).tolist()

    def run(graphs):
        engine = Engine(model, max_tokens=1024, n_slots=3, max_seq_len=256, use_graphs=graphs)
        a, b, c = slots = [engine.alloc_slot() for _ in range(3)]
        out = []

        def step(s, t):
            out.append(engine.step(s, t).clone())
        step(slots, [ids(70, 1), ids(9, 2), ids(33, 3)])
        for i in range(2):                       # the first of a size captures, the second replays
            step([a], [ids(20, 10 + i)])
            step([b, c], [ids(3, 20 + i), ids(2, 30 + i)])
            step(slots, [ids(1, 40 + i), ids(1, 50 + i), ids(1, 60 + i)])
            step([c], [ids(1, 70 + i)])
        torch.cuda.synchronize()
        engine.check_status()
        return out

    try:
        for graphs in (False, True):
            ops.launch_overlap(False)
            want = run(graphs)
            assert all(bool(torch.isfinite(x).all()) for x in want)
            ops.launch_overlap(True)
            for _ in range(2):
                got = run(graphs)
                assert all(torch.equal(x, y) for x, y in zip(got, want)), f"graphs {graphs}"
    finally:
        ops.launch_overlap(True)
