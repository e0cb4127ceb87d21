"""What a user of this package has it do, as measurable cases.

The package trains draft models against a verifier, so a case is one call of the work around that: an
optimizer step of one of the five algorithms (``Trainer.train_step``: forward, backward, clipping and the
optimizer), a validation batch (``Trainer.val_epoch``: forward only), or a forward of the verifier that
makes the hidden states a draft is trained on (``TensorParallelVerifier.forward``).  Widths are those of the
benchmark's and the examples' verifiers plus two generic ones (a plumbing size and a head dim of 64); rows are
packed from several documents of uneven length with a padded tail, as the collate function makes them; the
optimizers, losses and samplers are the command line's choices.  Everything computes in bf16 with fp32 state,
which is what the command line trains in on a GPU.

Weights are random at the initial scale, and the verifier's last states are drawn so that its
distribution over the draft vocabulary has a clear favourite in most rows, as a trained verifier's has.
"""

from __future__ import annotations

import math
import os
import tempfile

import torch

from speculators_b200.config import SpeculatorsConfig, VerifierConfig
from speculators_b200.layer_config import TransformerLayerConfig
from speculators_b200.models.dflash import DFlashDraftModel, DFlashSpeculatorConfig
from speculators_b200.models.dspark import DSparkDraftModel, DSparkSpeculatorConfig
from speculators_b200.models.eagle3 import Eagle3DraftModel, Eagle3SpeculatorConfig
from speculators_b200.models.mtp import MTPDraftModel, MTPSpeculatorConfig
from speculators_b200.models.peagle import PEagleDraftModel, PEagleSpeculatorConfig
from speculators_b200.proposals.greedy import GreedyTokenProposalConfig
from speculators_b200.train import Trainer, TrainerConfig
from speculators_b200.train.synthetic import SyntheticLoader
from speculators_b200.verifier.tp import TensorParallelVerifier

_LLAMA = {"architectures": ["LlamaForCausalLM"], "model_type": "llama", "rms_norm_eps": 1e-5, "rope_theta": 500000.0,
          "max_position_embeddings": 16384, "hidden_act": "silu"}
_QWEN3 = {"architectures": ["Qwen3ForCausalLM"], "model_type": "qwen3", "rms_norm_eps": 1e-6, "rope_theta": 1000000.0,
          "max_position_embeddings": 16384, "hidden_act": "silu"}

# Decoder widths by verifier: the benchmark's (8B, 70B, the mixture-of-experts head), the examples' 0.6B, the
# plumbing size, and a generic 2048-wide decoder with 64-wide heads.
_WIDTHS = {
    "tiny": dict(_LLAMA, hidden_size=256, num_hidden_layers=6, num_attention_heads=4, num_key_value_heads=2, head_dim=64,
                 intermediate_size=688, vocab_size=1024),
    "heads64_2k": dict(_LLAMA, hidden_size=2048, num_hidden_layers=16, num_attention_heads=32, num_key_value_heads=8, head_dim=64,
                       intermediate_size=8192, vocab_size=128256),
    "llama31_8b": dict(_LLAMA, hidden_size=4096, num_hidden_layers=32, num_attention_heads=32, num_key_value_heads=8, head_dim=128,
                       intermediate_size=14336, vocab_size=128256),
    "llama33_70b": dict(_LLAMA, hidden_size=8192, num_hidden_layers=80, num_attention_heads=64, num_key_value_heads=8, head_dim=128,
                        intermediate_size=28672, vocab_size=128256),
    "qwen3_0_6b": dict(_QWEN3, hidden_size=1024, num_hidden_layers=28, num_attention_heads=16, num_key_value_heads=8, head_dim=128,
                       intermediate_size=3072, vocab_size=151936),
    "qwen3_8b": dict(_QWEN3, hidden_size=4096, num_hidden_layers=36, num_attention_heads=32, num_key_value_heads=8, head_dim=128,
                     intermediate_size=12288, vocab_size=151936),
    "qwen3_next_mtp": dict(_QWEN3, architectures=["Qwen3NextForCausalLM"], model_type="qwen3_next", hidden_size=2048, num_hidden_layers=48,
                           num_attention_heads=16, num_key_value_heads=2, head_dim=256, intermediate_size=5632, vocab_size=151936,
                           rope_theta=10000000.0, partial_rotary_factor=0.25, num_experts=512, num_experts_per_tok=10,
                           moe_intermediate_size=512, shared_expert_intermediate_size=512, norm_topk_prob=True,
                           decoder_sparse_step=1, mlp_only_layers=[]),
}
_AUX = 3  # verifier layers whose states a draft reads
_WINDOW = 2048  # the command line's sliding window of a draft layer
_TTT = 3  # training-time-test passes of EAGLE-3, speculative steps of MTP


def listed():
    return [
        # the plumbing configuration of the tutorials and CPU tests: every launch counts
        _train("eagle3_tiny_128", "eagle3", "tiny", 128, documents=1, pad=0, draft_vocab=512, optimizer="adamw"),
        # a short ragged row at head dim 64
        _train("eagle3_heads64_1001", "eagle3", "heads64_2k", 1001, documents=3, pad=23, draft_vocab=32000, optimizer="adamw"),
        # the headline benchmark: one document of 2048 tokens for an 8B verifier
        _train("eagle3_8b_2048", "eagle3", "llama31_8b", 2048, documents=1, pad=0, draft_vocab=32000, optimizer="adamw"),
        # the command line's default flags: 8192 packed tokens, Muon
        _train("eagle3_8b_8192_muon", "eagle3", "llama31_8b", 8192, documents=11, pad=157, draft_vocab=32000, optimizer="muon"),
        # the widest draft the benchmark names
        _train("eagle3_70b_1536", "eagle3", "llama33_70b", 1536, documents=2, pad=10, draft_vocab=32000, optimizer="adamw"),
        # five-layer block drafter of the benchmark
        _train("dflash_8b_4096", "dflash", "qwen3_8b", 4096, documents=3, pad=0, draft_vocab=32000, optimizer="adamw", layers=5,
               block=16, anchors=512),
        # the 0.6B example: Markov and confidence heads, blocks of 8, default optimizer
        _train("dspark_0_6b_3000", "dspark", "qwen3_0_6b", 3000, documents=5, pad=61, draft_vocab=32000, optimizer="muon", layers=5,
               block=8, anchors=512),
        # the P-EAGLE example: 8 depths, trainable embeddings, row counts that change from step to step
        _train("peagle_8b_2048", "peagle", "qwen3_8b", 2048, documents=2, pad=0, draft_vocab=32000, optimizer="adamw", depths=8,
               anchors=2048),
        # fine-tuning a dense multi-token-prediction head over the verifier's full vocabulary
        _train("mtp_8b_2000", "mtp", "qwen3_8b", 2000, documents=1, pad=0, draft_vocab=151936, optimizer="adamw"),
        # the mixture-of-experts head of the benchmark with half of its experts (three states of it have to fit): head dim 256
        _train("mtp_moe_4096", "mtp", "qwen3_next_mtp", 4096, documents=1, pad=0, draft_vocab=151936, optimizer="adamw", experts=256),
        # a batch of the validation epoch
        _validate("validate_8b_5003", "llama31_8b", 5003, documents=7, pad=83, draft_vocab=32000),
        # hidden states of one prompt and response from the layers of an 8B verifier (what more layers do is the same again,
        # with more of a random decoder's rounding in it)
        _verify("verifier_8b_1777", "llama31_8b", 1777, layers=8),
    ]


def _train(name, algorithm, width, tokens, documents, pad, draft_vocab, optimizer, layers=1, block=0, anchors=0, depths=0, experts=0):
    return dict(name=name, path="train", algorithm=algorithm, width=width, tokens=tokens, documents=documents, pad=pad,
                draft_vocab=draft_vocab, optimizer=optimizer, layers=layers, block=block, anchors=anchors, depths=depths, experts=experts)


def _validate(name, width, tokens, documents, pad, draft_vocab):
    return dict(name=name, path="validate", algorithm="eagle3", width=width, tokens=tokens, documents=documents, pad=pad,
                draft_vocab=draft_vocab, optimizer="adamw", layers=1, block=0, anchors=0, depths=0, experts=0)


def _verify(name, width, tokens, layers):
    return dict(name=name, path="verifier", width=width, tokens=tokens, layers=layers)


def draw(rng):
    """One more case: any listed kind of work, sizes over the whole range that the listed ones span."""

    def log_int(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    def row(least, most):
        tokens = log_int(least, most)
        return dict(tokens=tokens, documents=rng.randint(1, max(1, min(12, tokens // 100))), pad=rng.choice([0, rng.randint(0, tokens // 16)]))

    optimizer = rng.choice(["adamw", "muon"])
    vocab = rng.choice([8000, 16000, 32000])
    kind = rng.choice(["eagle3", "eagle3", "eagle3", "eagle3_70b", "dflash", "dspark", "peagle", "mtp", "mtp_moe", "validate", "verifier"])
    if kind == "eagle3":
        width = rng.choice(["tiny", "heads64_2k", "qwen3_0_6b", "llama31_8b", "qwen3_8b"])
        c = _train("", "eagle3", width, **row(128, 4096 if width == "tiny" else 8192), draft_vocab=512 if width == "tiny" else vocab, optimizer=optimizer)
    elif kind == "eagle3_70b":
        c = _train("", "eagle3", "llama33_70b", **row(512, 1536), draft_vocab=vocab, optimizer="adamw")
    elif kind in ("dflash", "dspark"):
        width = rng.choice(["qwen3_0_6b", "qwen3_8b"])
        c = _train("", kind, width, **row(512, 4096), draft_vocab=vocab, optimizer="adamw" if width == "qwen3_8b" else optimizer,
                   layers=rng.randint(2, 5), block=rng.choice([8, 16]), anchors=log_int(64, 512))
    elif kind == "peagle":
        c = _train("", "peagle", rng.choice(["qwen3_0_6b", "qwen3_8b"]), **row(512, 2048), draft_vocab=vocab, optimizer="adamw",
                   depths=rng.randint(3, 8), anchors=2048)
    elif kind == "mtp":
        c = _train("", "mtp", rng.choice(["qwen3_0_6b", "qwen3_8b"]), tokens=log_int(256, 2048), documents=1, pad=0, draft_vocab=151936, optimizer="adamw")
    elif kind == "mtp_moe":
        c = _train("", "mtp", "qwen3_next_mtp", tokens=log_int(512, 4096), documents=1, pad=0, draft_vocab=151936, optimizer="adamw",
                   experts=rng.choice([64, 128, 256]))
    elif kind == "validate":
        c = _validate("", rng.choice(["heads64_2k", "qwen3_0_6b", "llama31_8b", "qwen3_8b"]), **row(256, 8192), draft_vocab=vocab)
    else:
        c = _verify("", rng.choice(["qwen3_0_6b", "heads64_2k", "llama31_8b", "qwen3_8b"]), log_int(64, 4096), layers=rng.randint(6, 9))
    del c["name"]
    return c


# --------------------------------------------------------------------------------------------------- preparation
def prepare(case, seed):
    """The trainer (or verifier) and one batch on the GPU."""
    torch.manual_seed(seed)  # initial weights here; the anchor and depth samplers of the steps draw from it too
    gen = torch.Generator(device="cuda").manual_seed(seed + 1)
    if case["path"] == "verifier":
        return _prepare_verifier(case, seed, gen)
    cfg = _layer_config(case)
    model, kwargs = _build(case, cfg)
    batch = _batch(case, cfg, model, gen)
    trainer = Trainer(model, TrainerConfig(
        lr=1e-4, muon_lr=1e-3, num_epochs=1, save_path=os.path.join(tempfile.gettempdir(), "sb200_cases_nothing_saved"),
        train_call_kwargs=kwargs, val_call_kwargs=kwargs, optimizer=case["optimizer"], scheduler_type="none", log_freq=10**9, device="cuda:0",
    ), SyntheticLoader([batch], 1), SyntheticLoader([batch], 1))
    trainer.model.train(case["path"] == "train")
    torch.manual_seed(seed)
    return {"case": case, "trainer": trainer, "batch": batch}


def _prepare_verifier(case, seed, gen):
    cfg = dict(_WIDTHS[case["width"]], num_hidden_layers=case["layers"])
    with torch.device("cuda"):
        verifier = TensorParallelVerifier(cfg, seed=seed, device="cuda", dtype=torch.bfloat16, resident=True)
        verifier.forward(torch.zeros(8, dtype=torch.long), [0])  # draws the weights and keeps them
    n, T = case["layers"], case["tokens"]
    return {"case": case, "verifier": verifier, "layer_ids": [2, n // 2, n - 3],
            "input_ids": torch.randint(0, cfg["vocab_size"], (1, T), generator=gen, device="cuda")}


def _layer_config(case):
    cfg = dict(_WIDTHS[case["width"]])
    if case["algorithm"] == "mtp":
        if case["experts"]:
            cfg["num_experts"] = case["experts"]
        return cfg
    # a window on every draft layer; the block drafters' first layer sees everything
    types = ["sliding_attention"] * case["layers"]
    if case["algorithm"] in ("dflash", "dspark"):
        types[0] = "full_attention"
    return dict(cfg, num_hidden_layers=case["layers"], sliding_window=_WINDOW, layer_types=types)


def _build(case, cfg):
    """The draft model with its frozen embedding and heads filled in, and what the trainer calls it with."""
    algorithm, vocab = case["algorithm"], case["draft_vocab"]
    layer = TransformerLayerConfig(**cfg)
    eagle = dict(norm_before_residual=True, norm_before_fc=True, norm_output=True, eagle_aux_hidden_state_layer_ids=[2, 5, 8])
    mask_token = cfg["vocab_size"] - 1
    with torch.device("cuda"):
        if algorithm == "eagle3":
            model = Eagle3DraftModel(Eagle3SpeculatorConfig(transformer_layer_config=layer, draft_vocab_size=vocab, **eagle))
            kwargs, _ = Eagle3DraftModel.get_trainer_kwargs(loss_fn="kl_div", ttt_steps=_TTT, ttt_step_loss_decay=1.0)
        elif algorithm == "peagle":
            model = PEagleDraftModel(PEagleSpeculatorConfig(transformer_layer_config=layer, draft_vocab_size=vocab, mask_token_id=mask_token, **eagle))
            kwargs, _ = PEagleDraftModel.get_trainer_kwargs(loss_fn="kl_div", num_depths=case["depths"], max_anchors=case["anchors"])
        elif algorithm == "dflash":
            model = DFlashDraftModel(DFlashSpeculatorConfig(transformer_layer_config=layer, draft_vocab_size=vocab, block_size=case["block"],
                                                            mask_token_id=mask_token, aux_hidden_state_layer_ids=[2, 5, 8]))
            kwargs, _ = DFlashDraftModel.get_trainer_kwargs(loss_fn="ce", per_position_loss_weight="dpace", max_anchors=case["anchors"])
        elif algorithm == "dspark":
            model = DSparkDraftModel(DSparkSpeculatorConfig(transformer_layer_config=layer, draft_vocab_size=vocab, block_size=case["block"],
                                                            mask_token_id=mask_token, aux_hidden_state_layer_ids=[2, 5, 8]))
            kwargs, _ = DSparkDraftModel.get_trainer_kwargs(loss_fn="kl_div", max_anchors=case["anchors"])
        else:
            model = MTPDraftModel(MTPSpeculatorConfig(transformer_layer_config=layer, speculators_config=SpeculatorsConfig(
                algorithm="mtp", proposal_methods=[GreedyTokenProposalConfig(speculative_tokens=_TTT)], default_proposal_method="greedy",
                verifier=VerifierConfig(name_or_path=None, architectures=cfg["architectures"]))))
            kwargs, _ = MTPDraftModel.get_trainer_kwargs(num_speculative_steps=_TTT)
        model.load_verifier_weights()  # no verifier on disk: leaves the tensors to be filled, drops what the algorithm has no use for
        with torch.no_grad():
            for name, p in model.named_parameters():
                if name.endswith("qkv_proj.weight"):  # scores of unit spread at every width, with or without head norms
                    p.normal_(0.0, p.shape[1] ** -0.5)
            model.embed_tokens.weight.normal_(0.0, 0.02)
            model.lm_head.weight.normal_(0.0, 0.02)
            if hasattr(model, "verifier_lm_head"):
                model.verifier_lm_head.weight.copy_(model.lm_head.weight)
        if model.use_draft_vocab:
            kept = torch.arange(vocab) * cfg["vocab_size"] // vocab
            t2d = torch.zeros(cfg["vocab_size"], dtype=torch.bool)
            t2d[kept] = True
            model.load_vocab_mappings(t2d, kept - torch.arange(vocab))
    return model, kwargs


def _batch(case, cfg, model, gen):
    """One packed row: uneven documents, a padded tail, supervised spans."""
    T, H = case["tokens"], cfg["hidden_size"]
    dev = "cuda"

    def normal(*shape):
        return torch.randn(*shape, generator=gen, device=dev)

    real = T - case["pad"]
    doc = torch.full((T,), -1, dtype=torch.long, device=dev)
    start = torch.zeros(T, dtype=torch.bool, device=dev)
    start[0] = True
    if case["documents"] > 1:
        start[1 + torch.randperm(real - 1, generator=gen, device=dev)[: case["documents"] - 1]] = True
    doc[:real] = torch.cumsum(start, 0)[:real] - 1
    at = torch.arange(T, device=dev)
    first = torch.cummax(torch.where(start, at, torch.zeros_like(at)), 0).values
    positions = torch.where(doc >= 0, at - first + (1 if case["algorithm"] in ("eagle3", "peagle") else 0), torch.zeros_like(at))
    mask = (torch.rand((T + 63) // 64, generator=gen, device=dev) < 0.6).repeat_interleave(64)[:T] & (doc >= 0)
    mask[real - 48 : real - 16] = True  # at least one answer, however short the row
    batch = {"input_ids": torch.randint(0, cfg["vocab_size"], (T,), generator=gen, device=dev), "loss_mask": mask, "position_ids": positions}
    if case["algorithm"] == "mtp":
        hs = normal(T, H)
        batch["hidden_states"] = hs / hs.pow(2).mean(-1, keepdim=True).sqrt()
    else:
        # the verifier's favourite token of each row: its last state leans towards that token's head row
        head = model.verifier_lm_head.weight
        liked = head[torch.randint(0, case["draft_vocab"], (T,), generator=gen, device=dev)].float()
        lean = min(1.0, 10.0 / (0.02 * H))
        batch["verifier_last_hidden_states"] = normal(T, H) + lean * math.sqrt(H) * liked / liked.norm(dim=-1, keepdim=True)
        batch["hidden_states"] = normal(T, _AUX * H)
        batch["document_ids"] = doc
    return {k: (v.to(torch.bfloat16) if v.is_floating_point() else v).unsqueeze(0) for k, v in batch.items()}


# --------------------------------------------------------------------------------------------------- one pass
def run(state):
    case = state["case"]
    if case["path"] == "verifier":
        return state["verifier"].forward(state["input_ids"], state["layer_ids"])
    trainer = state["trainer"]
    if case["path"] == "validate":
        # the accuracy counters beside the losses count hits of a random draft: a handful, and ties decide them
        return {k: v for k, v in trainer.val_epoch(0).items() if k.startswith("loss")}
    loss, _ = trainer.train_step(state["batch"])
    engine = trainer.engine
    out = {"loss": loss, "weights": engine.flat_w}
    if not case["experts"]:
        # With experts the gradients say which of two nearly equal experts a token went to: rounding decides that.
        out.update(gradients=engine.flat_g, first_moments=engine.exp_avg)
    return out


# --------------------------------------------------------------------------------------------------- work and tolerance
def work(case):
    cfg = _WIDTHS[case["width"]]
    H, hd, nh, nkv, inter = (cfg[k] for k in ("hidden_size", "head_dim", "num_attention_heads", "num_key_value_heads", "intermediate_size"))
    T = case["tokens"]
    layer = H * (nh + 2 * nkv) * hd + nh * hd * H + 3 * H * inter
    if case["path"] == "verifier":
        flops = case["layers"] * (2.0 * layer * T + 2.0 * T * T * nh * hd)
        return {"bytes": 2.0 * case["layers"] * layer + 2.0 * T * H * (1 + 4), "flops": flops}
    algorithm, V = case["algorithm"], case["draft_vocab"]
    doc = T / case["documents"]
    context = doc / 2 if doc <= _WINDOW else _WINDOW - _WINDOW**2 / (2 * doc)  # keys a query sees on average
    train = 3.0 if case["path"] == "train" else 1.0  # forward, input gradient, weight gradient
    head = 2.0 if case["path"] == "train" else 1.0  # frozen heads have no weight gradient
    attend = 3.5 if case["path"] == "train" else 1.0
    inputs = 2.0 * T * (_AUX + 1) * H + 25.0 * T
    frozen = 2.0 * V * H
    if algorithm in ("eagle3", "peagle"):
        wide = layer + H * (nh + 2 * nkv) * hd  # q | k | v read two states
        trained = wide + _AUX * H * H
        rows, passes = T, _TTT
        if algorithm == "peagle":
            seeds = 0.6 * T
            rows, passes = T + sum(int(seeds * max(0.7**d, 0.2)) for d in range(1, case["depths"])), 1
            trained += cfg["vocab_size"] * H
        flops = passes * rows * (2.0 * train * wide + 2.0 * head * V * H + attend * 4.0 * context * nh * hd)
        flops += rows * (2.0 * train * _AUX * H * H + 2.0 * V * H)
        frozen *= 2
    elif algorithm in ("dflash", "dspark"):
        n, L = case["anchors"] * case["block"], case["layers"]
        trained = L * layer + _AUX * H * H
        flops = 2.0 * train * (L * (n * layer + T * H * 2 * nkv * hd) + T * _AUX * H * H) + 2.0 * (head + 1) * n * V * H
        flops += L * attend * 4.0 * n * context * nh * hd
        frozen *= 2
        if algorithm == "dspark":
            trained += 256 * (cfg["vocab_size"] + V)
            flops += 2.0 * train * n * 256 * V
    else:
        if case["experts"]:
            q = 2 * nh * hd
            expert = 3 * H * cfg["moe_intermediate_size"]
            dense = H * (q + 2 * nkv * hd) + nh * hd * H + expert + H * case["experts"] + 2 * H * H
            trained, active = dense + case["experts"] * expert, dense + cfg["num_experts_per_tok"] * expert
        else:
            trained = active = layer + 2 * H * H
        flops = _TTT * T * (2.0 * train * active + 2.0 * head * V * H + attend * 4.0 * (T / 2) * nh * hd)
        inputs = 2.0 * T * H + 17.0 * T
    if case["path"] == "validate":
        return {"bytes": inputs + frozen + 2.0 * trained, "flops": flops}
    state = 32.0 * trained  # weights and gradients in bf16; master copy and two moments read and written
    if case["optimizer"] == "muon":
        # one moment; five iterations of a Gram matrix, its square (symmetric, both) and a product
        state = 24.0 * trained
        n_layers = case["layers"] if algorithm in ("dflash", "dspark") else 1
        q_in = 2 * H if algorithm in ("eagle3", "peagle") else H
        for m, n, times in (((nh + 2 * nkv) * hd, q_in, n_layers), (H, nh * hd, n_layers), (2 * inter, H, n_layers), (H, inter, n_layers), (H, _AUX * H, 1)):
            a, b = min(m, n), max(m, n)
            flops += times * 5 * (3.0 * a * a * b + 1.0 * a**3)
    return {"bytes": inputs + frozen + state, "flops": flops}


def tolerance(case):
    """bf16 products and activations with fp32 accumulation; a validation loss is an fp32 mean of them."""
    if case["path"] == "validate":
        return {"rel": 1e-3}
    if case["path"] == "verifier" or case["layers"] > 1:  # roundings of several layers add up
        return {"rel": 2.5e-2, "max": 0.9}
    return {"rel": 2e-2, "max": 0.9}
