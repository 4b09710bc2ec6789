"""Per-grid-shape launch tuning.

The marching stencil kernels give a warp a run ("chunk") of levels; how long
it should be depends on the grid: a large plane has rows enough to fill the
148 SMs with long chunks (each starts with its window's loads and its lower
face flux), a small plane needs short chunks to have warps enough at all.
The kernels choose a chunk themselves (0) by the number of rows.
``Autotuner`` times that and each fixed chunk once per (kernel, grid shape)
with CUDA events on the launching stream and keeps the fastest; the table can
be saved to and loaded from a JSON file so that a production run pays the
search once.
"""

from __future__ import annotations

import json
from pathlib import Path
from typing import Callable, Iterable

import torch

LEVEL_CHUNKS = (0, 1, 2, 4, 8, 16, 32, 64, 128)
# part of a table's keys: raised when the tuned kernels change, so that a saved
# table of other kernels is searched again
KERNELS = 2


class Autotuner:
    def __init__(self, path: str | Path | None = None, *, warmup: int = 2, repeats: int = 5):
        self.path = None if path is None else Path(path)
        self.warmup, self.repeats = warmup, repeats
        self.table: dict[str, dict] = {}
        if self.path is not None and self.path.exists():
            self.table = json.loads(self.path.read_text())

    @staticmethod
    def key(kind: str, ni: int, nj: int, nk: int) -> str:
        return f"{kind}@{KERNELS}:{ni}x{nj}x{nk}"

    def choose(self, kind: str, ni: int, nj: int, nk: int, run: Callable[[int], None],
               candidates: Iterable[int] = LEVEL_CHUNKS) -> int:
        """The fastest candidate for ``run(candidate)`` (one launch of the
        kernel with that setting on the current stream, 0 the kernel's own
        choice); cached per key.  The table holds it as "chosen", beside the
        fastest fixed candidate ("best")."""
        k = self.key(kind, ni, nj, nk)
        if k in self.table:
            return int(self.table[k]["chosen"])
        stream = torch.cuda.current_stream()
        times = {}
        for c in candidates:
            if c > nk:
                continue
            for _ in range(self.warmup):
                run(c)
            start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            start.record(stream)
            for _ in range(self.repeats):
                run(c)
            end.record(stream)
            end.synchronize()
            times[c] = start.elapsed_time(end) / self.repeats
        chosen = min(times, key=times.get)
        best = min((c for c in times if c), key=times.get, default=chosen)
        self.table[k] = {"best": best, "chosen": chosen, "ms": {str(c): t for c, t in times.items()}}
        return chosen

    def save(self) -> None:
        if self.path is not None:
            self.path.write_text(json.dumps(self.table, indent=1, sort_keys=True))


_default: Autotuner | None = None


def default_tuner() -> Autotuner:
    global _default
    if _default is None:
        _default = Autotuner()
    return _default
