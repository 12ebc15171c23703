"""B200-native Kimi Delta Attention prefill, behind the reference's `flash_kda.fwd` signature.

Python host side of the drop-in boundary: mirrors flash_kda/__init__.py:5-41 and the argument
checks of csrc/flash_kda.cpp:44-174 of the reference, then calls the C-ABI library
(include/fkda.h) with raw device pointers and torch's current CUDA stream: an ordinary call through a
small CPython extension (csrc/fkda_host.cpp), every other one, and all of them where that extension
does not fit the running torch, through ctypes.
There is no CPU or PyTorch fallback: without the compiled library, or without a CUDA device,
`fwd` raises.
"""
from ._binding import (FLAG_FUSED_ANY_T, FLAG_OPERANDS_PER_ITEM, FLAG_PREPARE_MMA_SYNC, FLAG_PREPARE_TCGEN05, FLAG_NO_FUSED_SHORT, FLAG_REFERENCE_ROUNDING, FLAG_SCAN_LOOKAHEAD, FLAG_SCAN_NO_SEGMENTS, FLAG_SCAN_PLAIN, FLAG_SCAN_SIMT, FLAG_SEGMENTS, fwd, get_workspace_size, last_error, lib, lib_path, operands, recurrence, recurrence_giveup,
                       plan_segments, prepare, prologue, read_status, scan, scan_giveup, prepare_giveup, selftest_umma, tmem_layout_probe, umma_bench, workspace_layout)

__all__ = ["fwd", "get_workspace_size", "prepare", "scan", "prologue", "read_status",
           "workspace_layout", "selftest_umma", "lib", "lib_path", "last_error", "FLAG_SCAN_SIMT", "FLAG_SCAN_PLAIN", "FLAG_SCAN_LOOKAHEAD",
           "FLAG_SCAN_NO_SEGMENTS", "FLAG_NO_FUSED_SHORT", "FLAG_REFERENCE_ROUNDING", "FLAG_SEGMENTS", "plan_segments", "tmem_layout_probe", "umma_bench", "scan_giveup", "prepare_giveup", "operands", "recurrence", "recurrence_giveup", "FLAG_FUSED_ANY_T", "FLAG_PREPARE_TCGEN05", "FLAG_PREPARE_MMA_SYNC", "FLAG_OPERANDS_PER_ITEM"]
