"""Decode sessions: CUDA-graph capture of the engine's per-step launch sequence and the public
generate loop.

`DecodeSession.generate()` is the user-facing call: prompt token ids in, generated ids out.  Each
decode step copies that step's inputs from pinned host memory, replays the captured graph and reads
the chosen tokens back (the tokens have to reach the host anyway to be streamed to a client).
`run_device_loop()` instead feeds the chosen token back on the device, so K steps are K graph replays
with no host round trip - the kernel-only number.

Reference behaviour being replaced: lazily captured per-shape CUDA graphs keyed by (rows, bindings)
(docs/ENGINEERING.md:23, rust/crates/ds41rt-daemon/src/v41_layer_graphs.rs).
"""
from __future__ import annotations

import array
import ctypes as C
from typing import Dict, List, Optional

import torch

from ..models.base import RowsEngine, whole_numbers
from ..ops import lib


class DecodeSession:
    def __init__(self, engine: RowsEngine, use_graphs: bool = True):
        self.e = engine
        self.use_graphs = use_graphs and engine.device.type == "cuda"
        self.graphs: Dict[tuple, torch.cuda.CUDAGraph] = {}
        self.launches_per_graph: Dict[tuple, int] = {}
        R = engine.max_rows
        # a step's inputs (tokens, positions, slots of its rows, one after the other) and its result
        self.h_in = torch.zeros(3 * R, dtype=torch.int32).pin_memory()
        self.h_chosen = torch.zeros(R, dtype=torch.int32).pin_memory()
        self._in, self._chosen = self.h_in.numpy(), self.h_chosen.numpy()
        self._view = memoryview(self._in)             # takes a list's numbers in a fifth of the array's time
        self.h2d_bytes = 0
        self.d2h_bytes = 0

    # ------------------------------------------------------------------ graphs
    def _enqueue(self, rows: int, feedback: bool):
        self.e.forward_rows(rows)
        if feedback:
            self.e._run("feedback", self.e.k.ds41_decode_feedback, lib.ptr(self.e.chosen), lib.ptr(self.e.in_tokens),
                        lib.ptr(self.e.row_pos), rows, lib.stream())

    def graph(self, rows: int, feedback: bool = False) -> Optional[torch.cuda.CUDAGraph]:
        key = (rows, feedback)
        if not self.use_graphs:
            return None
        if key not in self.graphs:
            before = self.e.launches
            self.graphs[key] = self.e.capture(lambda: self._enqueue(rows, feedback))
            self.launches_per_graph[key] = (self.e.launches - before) // 2      # an eager rehearsal, then the capture
        return self.graphs[key]

    # ------------------------------------------------------------------ stepping
    def step(self, tokens: List[int], positions: List[int], slots: List[int]) -> List[int]:
        """One pass through the public path: the inputs from pinned memory, graph replay, the result back into it."""
        n = len(tokens)
        e = self.e
        if not 0 < n <= e.max_rows:
            raise ValueError(f"a step has 1 to {e.max_rows} rows, not {n}")
        for i, values in enumerate((tokens, positions, slots)):
            try:
                self._view[i * n:(i + 1) * n] = array.array("i", values if type(values) is list else whole_numbers(values))
            except (TypeError, ValueError, OverflowError):       # other numbers, or one for all rows
                self._in[i * n:(i + 1) * n] = whole_numbers(values)
        self.h2d_bytes += 3 * 4 * n
        g = self.graph(n)
        src, dst, s = lib.ptr(self.h_in), lib.ptr(self.h_chosen), lib.stream()
        rows = (lib.ptr(e.in_tokens), lib.ptr(e.row_pos), lib.ptr(e.row_slot))
        if g is not None:
            lib.check(e.k.ds41_graph_step(C.c_void_p(g.raw_cuda_graph_exec()), src, *rows, lib.ptr(e.chosen), dst, n, s),
                      "decode step")
        else:
            lib.check(e.k.ds41_step_inputs(src, *rows, n, s), "step inputs")
            e.forward_rows(n)
            lib.check(e.k.ds41_step_result(lib.ptr(e.chosen), dst, n, s), "step result")
        self.d2h_bytes += 4 * n
        return self._chosen[:n].tolist()

    def run_device_loop(self, rows: int, steps: int):
        """`steps` decode steps with on-device token feedback (no host synchronisation inside)."""
        g = self.graph(rows, feedback=True)
        for _ in range(steps):
            if g is not None:
                g.replay()
            else:
                self._enqueue(rows, True)

    # ------------------------------------------------------------------ public generate
    def generate(self, prompt: List[int], max_new_tokens: int, slot: int = 0, eos: Optional[int] = None,
                 prefill_chunk: Optional[int] = None) -> List[int]:
        e = self.e
        assert e.cache.ensure(slot, len(prompt) + max_new_tokens + 1), "KV pool exhausted"
        nxt = e.prefill(slot, prompt, chunk=prefill_chunk)
        out = [nxt]
        pos = len(prompt)
        while len(out) < max_new_tokens and (eos is None or out[-1] != eos):
            out.append(self.step([out[-1]], [pos], [slot])[0])
            pos += 1
        e.check_status("generate")
        return out
