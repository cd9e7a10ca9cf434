"""What the captured steps with prompt portions are kept by (no GPU): steps that launch different things have different keys."""
from types import SimpleNamespace

import torch

from llm_serving_engine_b200.config.model_config import LayerSpec, ModelSpec, PartSpec
from llm_serving_engine_b200.models import DecoderModel, expected_tensors
from llm_serving_engine_b200.parts.attention import GroupedQueryAttention
from llm_serving_engine_b200.parts.base import Mixer
from llm_serving_engine_b200.parts.branches import ParallelMixers


def latent_model(windows, heads=16, rank=512, width=64, dtype=torch.bfloat16, device="cpu", scale=0.05, seed=0, positions=32768):
    """Latent attention layers alone, one per window."""
    norm = PartSpec("rmsnorm", {"eps": 1e-5})
    layers = tuple(LayerSpec(prefix=f"l{index}.", block=PartSpec("residual_streams", {"feed_forward": False}),
                             mixer=PartSpec("latent_attention", {"heads": heads, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": rank,
                                                                 "scale": scale, "eps": 1e-5, "window": window,
                                                                 "rot": {"base": 10000.0, "dims": 64}}),
                             feed_forward=None, mixer_norm=norm, feed_forward_norm=None) for index, window in enumerate(windows))
    spec = ModelSpec(architecture="latent layers", vocab_size=64, hidden_size=width, layers=layers, order=tuple(range(len(layers))),
                     final_norm=norm, embedding_name="embed", final_norm_prefix="final.", lm_head_name="head",
                     tie_word_embeddings=True, max_position_embeddings=positions)
    generator = torch.Generator().manual_seed(seed)
    weights = {}
    for name, tensor in expected_tensors(spec).items():
        values = torch.randn(tensor.shape, generator=generator)
        if tensor.kind == "matrix":
            weights[name] = (values * tensor.shape[-1] ** -0.5 * 1.5).to(dtype).to(device)
        else:
            weights[name] = (1.0 + 0.1 * values).to(device)
    return DecoderModel(spec, weights, dtype, device)


def test_a_layer_that_stops_expanding_its_latents_changes_the_key():
    """A windowed and a full layer: at 40,000 keys a request the full one's gathered rows would not fit, the windowed one's are as
    many as before."""
    model = latent_model([2048, 0])
    counts = [256] * 8
    short, long = (model.launch_signature(counts, [context] * 8) for context in (2304, 40000))
    rows = [[block.mixer._expanded_rows(counts, [context] * 8) for block in model.blocks] for context in (2304, 40000)]
    assert 2 * rows[0][0] * 576 <= 1 << 28      # bytes of gathered rows
    assert rows[0][0] == rows[0][1] == rows[1][0] > 0 and rows[1][1] == 0      # the layers' answers as a set are the same
    assert short != long
    assert model.launch_signature([256], [768]) != latent_model([0, 2048]).launch_signature([256], [20000])


def test_the_order_of_the_answers_is_part_of_the_key():
    a, b = latent_model([512, 0], heads=64), latent_model([0, 512], heads=64)
    for contexts in ([20000], [9000]):
        assert a.launch_signature([256], contexts) != b.launch_signature([256], contexts)


def test_a_long_prompt_in_portions_meets_few_classes():
    """Contexts of a prompt of 16,384 keys in portions of 512: at most two keys for every doubling, and room for all rows."""
    model = latent_model([0])
    mixer = model.blocks[0].mixer
    keys = set()
    for context in range(512, 16385, 512):
        key = model.launch_signature([512], [context])
        keys.add(key)
        rows, exact = mixer._expanded_rows([512], [context]), mixer._worth_expanding([512], [context])
        assert key == ((0, ("expanded", rows)),) and exact == context <= rows <= 1.5 * exact
    assert len(keys) <= 2 * 5 + 1


def test_scales_that_the_expanded_attention_refuses_go_over_the_latent_rows():
    """Its maximum is taken before the scale; over the latent rows any scale is taken, zero and negative ones too."""
    counts, contexts = [512], [512]
    for scale, expanded in ((0.05, True), (0.0, False), (-0.05, False)):
        assert (latent_model([0], scale=scale).blocks[0].mixer._expanded_rows(counts, contexts) > 0) == expanded, scale


def test_layers_without_an_answer_leave_the_key_empty():
    assert latent_model([0, 512]).launch_signature([1, 1], [700, 20]) == ()


def test_parallel_mixers_hand_on_what_their_branches_answer_at_their_contexts():
    class Branch(Mixer):
        def __init__(self, from_keys):
            self.from_keys = from_keys

        def launch_signature_at(self, segment_counts, contexts):
            return ("long",) if max(contexts) >= self.from_keys else ()

    part = object.__new__(ParallelMixers)
    part.branches = [Branch(100), Branch(1000)]
    answers = [part.launch_signature_at([8], [context]) for context in (50, 500, 5000)]
    assert answers[0] == () and len(set(answers)) == 3
    part.branches.reverse()
    assert part.launch_signature_at([8], [500]) != answers[1]      # another branch's answer


def test_general_attention_takes_few_rows_over_short_contexts_row_by_row():
    """The rule by rows and chunks at its edges, and that everything it follows from is in the key."""
    mixer = object.__new__(GroupedQueryAttention)
    mixer.head_dim, mixer.n_q, mixer.n_kv, mixer.window = 128, 12, 2, 0
    mixer.ctx = SimpleNamespace(dtype=torch.float32)

    def route(counts, contexts):
        signature = mixer.launch_signature_at(counts, contexts)
        longest = mixer._context_class(contexts)
        assert signature == ("general", *mixer._general_kernels(counts, longest), longest)
        return signature[1:3]

    assert route([64], [64]) == (False, False) and route([65], [65]) == (True, False)
    assert route([64], [256]) == (False, False) and route([64], [512]) == (True, False)      # 512 and 1,024 chunks
    assert route([8], [2048]) == (False, False) and route([10, 1], [2048, 5]) == (True, True)
    assert route([2] * 32, [4096] * 32) == (False, False) and route([2] * 33, [200] * 33) == (True, False)
    assert mixer.launch_signature_at([1, 1], [9, 9]) == ()
    mixer.head_dim = 192                                                                     # tiles take heads of up to 128
    assert route([500], [500]) == (False, False)
