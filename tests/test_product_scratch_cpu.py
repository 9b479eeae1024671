"""Scratch of the product-mode calls: two calls that run side by side share none of it."""
import torch


def test_two_calls_at_once_have_scratch_of_their_own():
    from spiky_b200.lut_data_manager import LUTDataManagerF

    dm = LUTDataManagerF(12, 8, 5, 4, 1, 2, 0, 32, 32)
    dm.register_synapse_meta(learning_rate=1.0, min_synaptic_weight=-1.0, max_synaptic_weight=1.0, initial_noise_level=0.0, initial_weight=0.0)
    dm.initialize_neurons(True)
    cfg, cpu = dm._cfg(0.0, sliced=False), torch.device("cpu")
    for backward in (False, True):
        (a, n), (b, m) = [dm._product_workspace(cfg, 3, 40, backward, 0, cpu) for _ in range(2)]
        assert n == m == a.numel() == b.numel() > 0
        assert a.data_ptr() + n <= b.data_ptr() or b.data_ptr() + m <= a.data_ptr()
