"""Named device buffers that live across steps.

Every intermediate of a step is a view of a buffer that was allocated once for the most
tokens a step may hold, so steady-state steps allocate nothing and a captured launch
sequence keeps reading and writing the same addresses.  ``version`` changes whenever a
buffer had to be replaced by a larger one; whoever captured addresses must capture again.

Beside these there is scratch that a faster way through a step takes and another way does without
(``spare``): it grows by doubling and stays within ``spare_bytes`` altogether.
"""

from __future__ import annotations


class Workspace:
    def __init__(self, device, min_rows: int = 1) -> None:
        self.device, self.min_rows = device, max(int(min_rows), 1)
        self._buffers: dict[str, object] = {}
        self._views: dict[tuple, tuple] = {}  # last view handed out per buffer
        self.version = 0
        self.spare_bytes: int | None = None  # what all spare scratch may take (None: whatever is asked for)
        self._spare: dict = {}  # its buffers' elements
        self._addressed: set = set()  # spare scratch whose addresses a capture may hold

    def buffer(self, name: str, rows: int, cols: int, dtype, rows_cap: int | None = 0):
        """A ``[rows, cols]`` view named ``name``.  Capacity is at least ``min_rows`` rows
        (``rows_cap=None``: exactly what is asked for, for buffers that are rarely large)."""
        key = (name, dtype)  # the same name may be wanted in two precisions by different paths
        hit = self._views.get(key)
        if hit is not None and hit[0] == rows and hit[1] == cols:
            return hit[2]  # the same view as last time: a step asks for every buffer once per layer
        import torch

        need = rows * cols
        buf = self._buffers.get(key)
        if buf is None or buf.numel() < need:
            cap_rows = rows if rows_cap is None else max(rows, self.min_rows, rows_cap)
            buf = torch.empty(max(cap_rows * cols, 1), dtype=dtype, device=self.device)
            if key in self._buffers:
                self.version += 1
            self._buffers[key] = buf
        view = buf[:need].view(rows, cols)
        self._views[key] = (rows, cols, view)
        return view

    def _spare_plan(self, wants):
        """Elements of each buffer that ``wants`` leads to (doubled where one grows, if that much may be taken), or None."""
        held = self._spare
        if all(held.get((name, dtype), -1) >= rows * cols for name, rows, cols, dtype in wants):
            return held
        for grown in (lambda n: 1 << max(n - 1, 0).bit_length(), int):
            plan = dict(held)
            for name, rows, cols, dtype in wants:
                if plan.get((name, dtype), -1) < rows * cols:
                    plan[name, dtype] = grown(max(rows * cols, 1))
            if self.spare_bytes is None or sum(n * dtype.itemsize for (_, dtype), n in plan.items()) <= self.spare_bytes:
                return plan
        return None

    def has_spare(self, wants) -> bool:
        """Whether :meth:`spare` would hand out ``wants``."""
        return self._spare_plan(wants) is not None

    def spare(self, wants, captured: bool = True):
        """``[rows, cols]`` views of spare scratch for ``wants`` (name, rows, cols, dtype), or None where that would be more than
        ``spare_bytes``.  ``captured=False``: scratch of steps that are launched one kernel at a time alone, whose growth
        leaves captured addresses as they are."""
        import torch

        captured = captured or (str(self.device).startswith("cuda") and torch.cuda.is_current_stream_capturing())
        plan, views = None, []
        for name, rows, cols, dtype in wants:
            key = (name, dtype)
            if captured:
                self._addressed.add(key)
            hit = self._views.get(key)
            if hit is not None and hit[0] == rows and hit[1] == cols:
                views.append(hit[2])
                continue
            if plan is None:
                plan = self._spare_plan(wants)
                if plan is None:
                    return None
            need = rows * cols
            buf = self._buffers.get(key)
            if buf is None or buf.numel() < need:
                if buf is not None and key in self._addressed:
                    self.version += 1
                self._views.pop(key, None)
                buf = self._buffers.pop(key, None)
                del buf  # (given back first: the larger one may need its place)
                buf = self._buffers[key] = torch.empty(plan[key], dtype=dtype, device=self.device)
                self._spare[key] = plan[key]
            view = buf[:need].view(rows, cols)
            self._views[key] = (rows, cols, view)
            views.append(view)
        return views

    def bytes(self) -> int:
        return sum(b.numel() * b.element_size() for b in self._buffers.values())
