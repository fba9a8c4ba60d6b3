"""leopard_b200 — B200-native (sm_100a) implementation of Leopard's multi-image prefill hot path.

Host code is Python/PyTorch (device memory, streams, torch.distributed); all arithmetic on the path runs in the
hand-written CUDA library `lib/libleopard_b200.so` behind the C ABI in `include/leopard_b200.h`.
The reference's scripts bind to it through hf.py, megatron.py and idefics2.py.
"""
__version__ = "0.1.0"
