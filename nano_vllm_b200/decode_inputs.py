"""Decode-step inputs in one launch.

Host mirror of what nano-vllm's ``ModelRunner`` does before it can replay a decode graph:
``prepare_decode`` / ``prepare_block_tables`` / ``prepare_sample``
(nanovllm/engine/model_runner.py:151-159, 218-258: six ``torch.tensor(..., pin_memory=True)
.cuda()`` round trips) and the clear-and-copy of the graph's static tensors in ``run_model``
(model_runner.py:271-282: five ``zero_()`` and five slice copies).  Here the step is packed into
one pinned staging block, which one launch (``nvllm_decode_step_inputs_pinned``) reads and expands
straight into the static tensors.

Staging block for a batch of n sequences (byte offsets)::

    0            tokens        int64[n]    last token of each sequence
    8n           lens          int32[n]    sequence length (the new token included)
    12n          temperatures  fp32[n]     read by the sampler, not by the kernel
    16n          offsets       int32[n+1]  prefix sum of the block-table lengths
    16n+4(n+1)   blocks        int32[...]  the block tables, concatenated
"""
from __future__ import annotations

import numpy as np
import torch

from . import _lib


def layout(n: int) -> dict[str, int]:
    """Byte offsets of the sections of the staging block for n sequences."""
    return {"tokens": 0, "lens": 8 * n, "temperatures": 12 * n, "offsets": 16 * n, "blocks": 16 * n + 4 * (n + 1)}


def staging_bytes(max_bs: int, table_width: int) -> int:
    return layout(max_bs)["blocks"] + 4 * max_bs * table_width


def pack(seqs, buf: np.ndarray, with_temperatures: bool = True, temperatures=None) -> tuple[int, int]:
    """Writes the step of ``seqs`` (objects with ``last_token``, ``num_tokens``, ``block_table``
    and, when ``with_temperatures``, ``temperature``: nanovllm/engine/sequence.py) into ``buf``
    (uint8).  Returns (bytes used, widest block table).  Tensor-parallel worker ranks pass
    ``with_temperatures=False``: the sequences they receive carry no sampling parameters
    (Sequence.__getstate__, sequence.py:74-76) and only rank 0 samples -- unless the caller
    hands the step's ``temperatures`` over as a list (the vocabulary-sharded sampling step)."""
    return _lib.host().pack(seqs, buf, with_temperatures, temperatures)


class DecodeInputStager:
    """Owns the pinned staging blocks and the device temperatures of one model runner.  The kernel reads
    the host block itself over PCIe (14 KB at batch 256), so a step is one launch and no copy."""

    def __init__(self, max_bs: int, table_width: int, device):
        self.max_bs, self.table_width = max_bs, table_width
        nbytes = (staging_bytes(max_bs, table_width) + 15) // 16 * 16
        # two host blocks used in turn, each guarded by the event of the launch that last read it
        self.host = [torch.empty(nbytes, dtype=torch.uint8, pin_memory=True) for _ in range(2)]
        self.temperatures = torch.empty(max_bs, dtype=torch.float32, device=device)
        self._native = _lib.host()
        self._state = self._native.make_stager(*self.host, self.temperatures, max_bs, table_width)

    def stage(self, seqs, graph_bs: int, graph_vars: dict, with_temperatures: bool = True,
              temperatures=None) -> torch.Tensor:
        """Fills rows [0, graph_bs) of ``graph_vars`` (the runner's static input tensors,
        model_runner.py:302-307) for a decode step of ``seqs``; returns the step's temperatures
        as a device tensor.  Everything is enqueued on the current stream."""
        return self._native.stage(self._state, seqs, graph_bs, with_temperatures, temperatures, graph_vars["input_ids"],
                                  graph_vars["positions"], graph_vars["slot_mapping"], graph_vars["context_lens"],
                                  graph_vars["block_tables"])
