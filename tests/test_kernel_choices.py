"""The runtime's choices of how to cut the work (K parts of a few-token product, key splits of decode
attention): what they may depend on, their bounds, and the cases that were measured."""
import pytest


def test_key_splits_depend_on_the_bucket_and_the_context_class_only():
    from odin_infer_b200.engine.runtime import context_class_of, decode_key_splits
    for n_seqs in (1, 2, 3, 4, 8, 12, 16, 24, 32, 64, 200, 256):
        for n_kv in (1, 2, 8):
            by_class = {}
            for longest in list(range(1, 1300, 37)) + [2048, 4000, 8192, 20000, 32768, 40000]:
                s = decode_key_splits(n_seqs, n_kv, longest)
                assert 1 <= s <= 16
                # never more CTAs than fit the GPU twice, unless one split already is
                assert s == 1 or n_seqs * n_kv * s <= 2 * 148
                cls = context_class_of(longest)
                assert by_class.setdefault(cls, s) == s, (n_seqs, n_kv, longest)


def test_key_splits_of_the_measured_cases():
    from odin_infer_b200.engine.runtime import decode_key_splits
    assert decode_key_splits(8, 8, 520) == 4       # 8 sequences of ~520 tokens: four splits were fastest
    assert decode_key_splits(4, 8, 520) == 4
    assert decode_key_splits(12, 8, 520) == 1      # from 12 sequences on: one
    assert decode_key_splits(16, 8, 520) == 1
    assert decode_key_splits(64, 8, 640) == 1
    assert decode_key_splits(4, 8, 32768) == 9     # long contexts: as many as fit the GPU twice
    assert decode_key_splits(1, 8, 32768) == 16
    assert decode_key_splits(3, 8, 100) == 1       # a page or two: nothing to split


def test_k_parts_fill_whole_rounds_and_never_depend_on_the_tokens():
    from odin_infer_b200.engine.runtime import choose_k_split
    # the 8B shape's decode products: q|k|v 48 tiles, o and down 32, gate|up 192; K blocks 64 or 192
    assert choose_k_split(48, 64, 8) == 3          # 144 CTAs
    assert choose_k_split(32, 64, 8) == 4          # 128
    assert choose_k_split(192, 64, 8) == 3         # 576 items, four rounds of 148
    assert choose_k_split(32, 192, 8) == 4
    for tiles in (1, 7, 32, 48, 100, 192, 1187):
        for kb in (1, 3, 16, 64, 192):
            for m in (1, 8, 16, 64, 128):
                s = choose_k_split(tiles, kb, m)
                assert 1 <= s <= 16 and s <= max(1, kb)
                per = (kb + s - 1) // s
                assert (kb + per - 1) // per == s, "an empty part"


def test_contexts_of_the_32_bit_path_are_one_class():
    import torch
    from odin_infer_b200.engine.runtime import Runtime, context_class_of
    lengths = (1, 511, 512, 513, 5000)
    assert len({Runtime("cpu", torch.float32).context_class(n) for n in lengths}) == 1
    assert [Runtime("cpu", torch.bfloat16).context_class(n) for n in lengths] == [context_class_of(n) for n in lengths]


def _model(raw):
    from odin_infer_b200.config import config_from_dict
    from odin_infer_b200.config.registry import lookup_architecture
    from odin_infer_b200.engine.model import DecoderModel
    model = DecoderModel(lookup_architecture(raw.get("architectures", [raw.get("architecture")])[0]).build_spec(config_from_dict(raw)))
    for pe in model.position_encodings.values():
        pe.cos = pe.sin = None   # (tables of a loaded model)
    return model


def _qwen3(heads, kv, head_dim):
    return dict(architectures=["Qwen3ForCausalLM"], hidden_size=256, intermediate_size=256, num_hidden_layers=2, num_attention_heads=heads,
                num_key_value_heads=kv, head_dim=head_dim, vocab_size=256, rope_theta=1e4, rms_norm_eps=1e-6, tie_word_embeddings=True)


def test_graphs_of_short_contexts_only_where_their_kernel_runs(monkeypatch):
    """A decode step has a graph of its own for short contexts exactly where a layer's attention launches another kernel for them."""
    import torch
    from odin_infer_b200.engine.runtime import Runtime
    from odin_infer_b200.parts.base import Mixer
    from odin_infer_b200.parts.state_space import SideBySide
    rt, f32 = Runtime("cpu", torch.bfloat16), Runtime("cpu", torch.float32)
    for heads, kv, hd in ((16, 8, 128), (8, 8, 64), (4, 2, 64)):
        assert _model(_qwen3(heads, kv, hd)).short_context(rt, 1) == 128
        assert _model(_qwen3(heads, kv, hd)).short_context(f32, 1) == 0
    for heads, kv, hd in ((4, 2, 32), (4, 2, 256), (34, 2, 64)):   # no tensor-core decode attention
        assert _model(_qwen3(heads, kv, hd)).short_context(rt, 1) == 0
    side = SideBySide.__new__(SideBySide)   # attention beside another mixer in one layer
    side.left, side.right = _model(_qwen3(16, 8, 128)).layers[0].mixer, Mixer()
    assert side.short_context(rt, 1) == 128
    for n_seqs in (1, 64, 256):
        assert _model(_qwen3(16, 8, 128)).short_context(rt, n_seqs) == 128   # one key split, whatever the batch
    monkeypatch.setenv("ODIN_DECODE_SPLITS", "2")
    assert _model(_qwen3(16, 8, 128)).short_context(rt, 1) == 0
    monkeypatch.delenv("ODIN_DECODE_SPLITS")
    monkeypatch.setenv("ODIN_FUSED_ATTENTION", "0")
    assert _model(_qwen3(16, 8, 128)).short_context(rt, 1) == 0


def test_the_table_of_streams_is_bounded(monkeypatch):
    """A program that makes streams without end gets the right one each time, and the table does not grow with them."""
    import torch
    from odin_infer_b200.csrc import ops
    now = [0]
    monkeypatch.setattr(ops, "_streams", {})
    monkeypatch.setattr(ops, "_current_raw_stream", lambda device: now[0])
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda: ("stream", now[0]))
    monkeypatch.setattr(torch._C, "_cuda_getCurrentStream", lambda device: (now[0], device, 1), raising=False)
    for now[0] in [*range(1000), *range(1000)]:
        assert ops.current_stream() == ("stream", now[0])
        assert len(ops._streams) <= 256
