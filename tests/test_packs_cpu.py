"""Pack tuples of a model on the CPU: which slots a step may leave empty."""
import torch

import hf_adapter_b200 as hb


def test_only_slots_that_a_step_does_not_read_are_left_empty():
    cfg = hb.NativeRWKV7Config(vocab_size=16, hidden_size=64, num_hidden_layers=3, num_heads=1, head_dim=64, intermediate_size=128,
                               decay_low_rank_dim=8, a_low_rank_dim=8, v_low_rank_dim=8, gate_low_rank_dim=8)
    m = hb.RWKV7ForCausalLM(cfg)
    del m.model.layers[2].attn.v_lora  # its gate is then the one of zero weights, in either form of the packs
    step, full = (hb.extract_graph_packs(m, unused_as_zeros=z)[0] for z in (False, True))
    none = [[j for j, v in enumerate(p) if v is None] for p in step]
    assert none == [[30, 31, 32], [5, 6], [5, 6]]  # layer 0's v LoRA; the pre-norm of the others
    for a, b in zip(step, full):
        assert all(x is None or not torch.is_tensor(x) or torch.equal(x, y) for x, y in zip(a, b))
    assert not any(v is None for p in full for v in p)


def test_dense_products_that_stay_on_the_library():
    from hf_adapter_b200.rows import prefers_dense
    # (rows, K, N, fused, early): each pair is the two sides of a line
    for take, leave in [((4, 256, 2048, False, False), (4, 248, 2048, False, False)), ((8, 256, 2048, True, False), (8, 248, 2048, True, False)),
                        ((1, 2560, 4096, False, False), (1, 2560, 4104, False, False)), ((1, 1024, 8192, False, False), (1, 1024, 8200, False, False)),
                        ((8, 4096, 8192, True, False), (8, 4104, 8192, True, False)), ((8, 4096, 16384, True, True), (8, 4104, 16384, True, True)),
                        ((8, 768, 16384, True, True), (8, 768, 16392, True, True)), ((1, 16384, 4096, True, False), (1, 20480, 5120, True, True))]:
        assert prefers_dense(*take) and not prefers_dense(*leave)


def test_quantised_products_on_the_row_kernel():
    from hf_adapter_b200.quant import few_rows_quant
    for K, N, most in [(128, 24, 8), (128, 16, 0), (7168, 4096, 8), (7296, 4096, 7), (8192, 1032, 7), (8320, 8192, 5), (12288, 8192, 5), (12416, 8192, 3),
                       (16384, 4096, 3), (12288, 1024, 0)]:
        assert [m for m in range(10) if few_rows_quant(m, K, N)] == list(range(1, most + 1))


def test_quantised_products_of_few_channels_on_the_row_kernel():
    from hf_adapter_b200.quant import few_rows_quant
    for K, N, bits, most in [(10240, 2560, 4, 3), (10240, 2560, 8, 5), (10240, 2568, 4, 5), (8192, 2056, 4, 7), (8200, 2056, 4, 5), (8320, 2064, 4, 3),
                             (8320, 2048, 4, 5), (12288, 2048, 4, 5), (16384, 4096, 8, 3)]:
        assert [m for m in range(10) if few_rows_quant(m, K, N, bits)] == list(range(1, most + 1)), (K, N, bits)
