"""What a step hands to the parts: the flattened batch and scratch memory.

All tokens of a step form one batch of T rows.  For row t: ``token_ids[t]``,
its absolute position in its request ``positions[t]``, and ``token_item[t]``,
the index of its entry in the step (the row of every block table).  These and
the block tables lie in one device buffer that is written with one copy per
step (the reference's ``BatchControl`` idea, engine/src/gpt2_gpu_batch.cu:18-24,
91-113); kernels read everything from there.
"""

from __future__ import annotations

import numpy as np
import torch

from ..kernels import ops


class Workspace:
    """Named scratch tensors, reused across layers and steps.  A buffer is
    allocated with room for ``min_rows`` rows and grows when a step needs more."""

    def __init__(self, device, min_rows: int):
        self.device = device
        self.min_rows = int(min_rows)
        self._buffers = {}
        self.generation = 0          # grows whenever a buffer moves (captured graphs are then stale)

    def get(self, tag: str, shape, dtype):
        rows, rest = int(shape[0]), tuple(int(s) for s in shape[1:])
        key = (tag, dtype, rest)
        held = self._buffers.get(key)
        if held is None or held.shape[0] < rows:
            capacity = max(rows, self.min_rows if held is None else 2 * held.shape[0])
            if tag == "logits":
                capacity = rows if held is None else max(rows, held.shape[0])
            # zeros, not whatever the memory held: rows that a step's kernels leave unwritten (tokens that fill a step
            # up to a round shape and are no tile's) are read by the kernels after them, and must be finite
            held = torch.zeros((capacity, *rest), dtype=dtype, device=self.device)
            self._buffers[key] = held
            self.generation += 1
        return held[:rows]


class ControlBlock:
    """The step's token arrays and block tables in one int32 device buffer, written with a
    single copy from pinned host memory.

    There are two device buffers.  Steps that ask for it (``alternate``) use them in turn and
    copy on a stream of their own: the arrays of step k+1 are on the device while the kernels
    of step k still read theirs, so no copy stands between two steps' kernels; a step's kernels
    wait for their copy, and a copy waits for the kernels that read the buffer it overwrites
    (``consumed`` records them).  Other steps keep to the first buffer (their kernels are
    replayed from graphs with fixed addresses): the host fills the parts of a ring in turn, and a step's
    first kernel (``take``) brings the part whose turn it is, which it counts on the device, into the buffer."""

    RING = 3                                  # parts: the host fills one while two steps are on their way

    def __init__(self, device, groups):
        self.device = device
        self.groups = [(g.index, g.max_blocks) for g in groups if g.paged]
        self.capacity = 0
        self.device_buffers = [None, None]
        self.copy_stream = torch.cuda.Stream(device=device)
        self._layouts = {}
        self._host_views = {}
        self.parity = 0
        self.generation = 0
        self.last_upload_bytes = 0            # bytes of the last step's host-to-device copy
        self.done = None                      # the event behind the last step's kernels (``consumed``)

    @staticmethod
    def tile_ints(n_tokens: int, n_items: int) -> int:
        """Room for the attention work list: at most n_tokens // 128 + n_items tiles, each in
        at most 8 parts, 8 int32 per record."""
        return 8 * 8 * (n_tokens // 128 + n_items)

    def _layout(self, n_tokens: int, n_items: int):
        """Offsets (in int32 units) as a function of the step's sizes only, so
        that steps of equal sizes find their arrays at equal addresses."""
        offsets = {"turn": 0}                     # the step's number modulo two: where its draws go on the host
        cursor = 4
        for name in ("token_ids", "positions", "token_item", "want_rows", "want_slots", "counters", "temperature",
                     "top_p"):
            offsets[name] = cursor
            cursor += n_tokens
        cursor += cursor & 1                      # 8-byte alignment for the 64-bit seeds
        offsets["seeds"] = cursor
        cursor += 2 * n_tokens
        offsets["att_tiles"] = cursor             # work list of the prompt-attention kernel
        cursor += self.tile_ints(n_tokens, n_items)
        for index, max_blocks in self.groups:
            offsets[("block_table", index)] = cursor
            cursor += n_items * max_blocks
        # per entry: its slot, the row of its first token, its tokens, the position of its first token
        for name in ("item_slot", "item_offset", "item_count", "item_start"):
            offsets[name] = cursor
            cursor += n_items
        return offsets, cursor

    def _ensure(self, size: int):
        if size <= self.capacity:
            return
        torch.cuda.synchronize(self.device)      # nothing may still read or fill the old buffers
        self.capacity = (max(size, 2 * self.capacity, 4096) + 3) // 4 * 4
        self.device_buffers = [torch.zeros(self.capacity, dtype=torch.int32, device=self.device) for _ in range(2)]
        self._host = [torch.zeros(self.capacity, dtype=torch.int32).pin_memory() for _ in range(2)]
        self._host_np = [h.numpy() for h in self._host]
        self._copied = [torch.cuda.Event(), torch.cuda.Event()]       # the copy out of host buffer t is done
        self._copied_once = [False, False]
        self._host_turn = 0
        self._consumed_by = [torch.cuda.Event(), torch.cuda.Event()]
        self._consumed = [None, None]        # the event behind the kernels that read device buffer p, once there are any
        self._ring = torch.zeros(self.RING * self.capacity, dtype=torch.int32).pin_memory()
        self._ring_np = self._ring.numpy()
        self._ring_address = ops.device_address(self._ring)
        self._ring_done = [torch.cuda.Event() for _ in range(self.RING)]      # the step that took part r is done
        self._ring_used = [False] * self.RING
        self._ring_turn, self._ring_open = 0, False
        self._steps = torch.zeros(2, dtype=torch.int32, device=self.device)
        self._layouts = {}                   # (parity, tokens, entries) -> (offsets, size, device views)
        self._host_views = {}                # (ring or not, part, tokens, entries) -> host views
        self.generation += 1

    def begin(self, n_tokens: int, n_items: int, alternate: bool = True):
        """The arrays of a step of these sizes: (host views to fill, device views).  ``send`` follows; until then nothing has
        changed: a step that is given up while its arrays are filled leaves no trace, and the next one begins where it did."""
        parity = (self.parity ^ 1) if alternate else 0
        key = (parity, n_tokens, n_items)
        held = self._layouts.get(key)
        if held is None:
            offsets, size = self._layout(n_tokens, n_items)
            size = (size + 3) // 4 * 4
            self._ensure(size)               # may drop every cached layout
            held = self._layouts[key] = (offsets, size, self._views(self.device_buffers[parity], offsets, n_tokens, n_items))
        offsets, size, views = held
        if alternate:
            # two pinned buffers in turn; the copy that last read this one must be done
            part = self._host_turn ^ 1
            if self._copied_once[part]:
                self._copied[part].synchronize()
        else:
            if self._ring_open:
                # a step was sent and did not get behind its kernels: whether they took its part is not known
                torch.cuda.synchronize(self.device)
                self._steps.zero_()
                torch.cuda.synchronize(self.device)
                self._ring_turn, self._ring_open = 0, False
            part = self._ring_turn
            if self._ring_used[part]:
                self._ring_done[part].synchronize()
        host_key = (alternate, part, n_tokens, n_items)
        host = self._host_views.get(host_key)
        if host is None:
            if len(self._host_views) >= 512:
                self._host_views.clear()
            memory = self._host_np[part] if alternate else self._ring_np[part * self.capacity:(part + 1) * self.capacity]
            host = self._host_views[host_key] = self._array_views(memory, offsets, n_tokens, n_items)
        self._begun = (parity, part, size)
        return host, views

    def send(self, alternate: bool = True) -> None:
        """The filled arrays are on their way (the alternating steps' copy), or ready to be taken (``take``)."""
        parity, turn, size = self._begun
        self.parity, self._size = parity, size
        self.last_upload_bytes = 4 * size
        if not alternate:
            self._ring_open = True
            return
        self._host_turn = turn
        # beside the kernels of the step before; behind the kernels that last read this buffer
        with torch.cuda.stream(self.copy_stream):
            if self._consumed[parity] is not None:
                self.copy_stream.wait_event(self._consumed[parity])
            self.device_buffers[parity][:size].copy_(self._host[turn][:size], non_blocking=True)
            self._copied[turn].record(self.copy_stream)
        torch.cuda.current_stream(self.device).wait_event(self._copied[turn])
        self._copied_once[turn] = True

    def take(self) -> None:
        """Launch the kernel that brings the step's arrays into the device buffer (the step's upload, which the count of the
        model's kernels leaves out as it left out the copy)."""
        ops.control(self.device_buffers[0], self._ring_address, self.capacity, self.RING, self._steps, self._size)

    def consumed(self, alternate: bool) -> None:
        """Call after the step's kernels are enqueued: its buffer may be overwritten once they
        are done."""
        compute = torch.cuda.current_stream(self.device)
        if alternate:
            self.done = self._consumed_by[self.parity]
        else:
            part = self._ring_turn
            self.done = self._ring_done[part]
            self._ring_used[part] = True
            self._ring_turn, self._ring_open = (part + 1) % self.RING, False
        self.done.record(compute)
        self._consumed[self.parity] = self.done

    def _array_views(self, memory, offsets, n_tokens: int, n_items: int):
        """The same as ``_views``, of the host's memory, as arrays of the types that are written."""
        views = {}
        for name, start in offsets.items():
            if name == "turn":
                views[name] = memory[start:start + 1]
            elif name == "seeds":
                views[name] = memory[start:start + 2 * n_tokens].view(np.uint64)
            elif name in ("temperature", "top_p"):
                views[name] = memory[start:start + n_tokens].view(np.float32)
            elif name == "att_tiles":
                views[name] = memory[start:start + self.tile_ints(n_tokens, n_items)].reshape(-1, 8)
            elif isinstance(name, tuple):
                views[name] = memory[start:start + n_items * dict(self.groups)[name[1]]].reshape(n_items, -1)
            elif name.startswith("item_"):
                views[name] = memory[start:start + n_items]
            else:
                views[name] = memory[start:start + n_tokens]
        return views

    def _views(self, buffer, offsets, n_tokens: int, n_items: int):
        views = {}
        for name, start in offsets.items():
            if name == "turn":
                views[name] = buffer[start:start + 1]
            elif name == "seeds":
                views[name] = buffer[start:start + 2 * n_tokens].view(torch.int64)
            elif name in ("temperature", "top_p"):
                views[name] = buffer[start:start + n_tokens].view(torch.float32)
            elif name == "att_tiles":
                views[name] = buffer[start:start + self.tile_ints(n_tokens, n_items)]
            elif isinstance(name, tuple):
                max_blocks = dict(self.groups)[name[1]]
                views[name] = buffer[start:start + n_items * max_blocks].view(n_items, max_blocks)
            elif name.startswith("item_"):
                views[name] = buffer[start:start + n_items]
            else:
                views[name] = buffer[start:start + n_tokens]
        return views


class StepContext:
    """The batch of one step, as the parts see it."""

    def __init__(self, kernels, workspace, act_dtype, device):
        self.kernels = kernels
        self.workspace = workspace
        self.act_dtype = act_dtype
        self.device = device
        self.n_tokens = 0
        self.n_items = 0
        self.n_want = 0
        self.token_ids = self.positions = self.token_item = self.want_rows = self.want_slots = None
        self.any_previous = False     # some token id is negative: -1 - slot names that slot's last sampled token
        self.item_slots = []          # host: slot of each entry
        self.item_starts = []         # host: position of each entry's first token
        self.item_counts = []         # host: tokens of each entry
        self.item_offsets = []        # host: row of each entry's first token
        self.item_slot = self.item_offset = self.item_count = self.item_start = None    # the same, on the device (int32)
        self.kept_results = None      # fp32 [T, planes, width]: the embedding output and every layer's result, if the model keeps them
        self.streams = None           # fp32 [T, streams, width]: the residual of a model with several residual streams
        self.next_norm = None         # the norm that reads the stream first in the next run entry, where it is known
        self.normed_ahead = None      # (that norm, its rows) once a pass over the stream has applied it
        self.streams_pending = None   # a layer's last write onto the streams, waiting to go with the next read-out
        self.in_ring = False          # the step's arrays come from the ring of control blocks, by the step's first kernel
        self.turn = None              # device int32 [1]: the step's number modulo two, where its draws go on the host
        self.steps_apart = False      # no kernel of an earlier step still runs when this step's kernels start, but for its first one: what
                                      # earlier steps left (cached rows, states) may be read ahead of the wait for the kernels ahead
        self.decode_only = False      # every entry brings exactly one token
        self.fused = False            # the step goes to the one-kernel decode step
        self.dump = None              # a list: the model appends the residual stream after every run entry
        self.att_tiles = None         # device work list (tiles of up to 128 tokens of one entry), or None
        self.n_att_tiles = 0          # records (CTAs) of the work list
        self.n_att_singles = 0        # the last ones of them: tokens that stand alone beside prompt portions
        self.n_split_tiles = 0        # tiles among them that come in several parts
        self.att_parts = 1            # most parts of a tile
        self.att_units = False        # the work list holds units of up to 256 tokens (two tiles) instead of tiles

    def buffer(self, tag: str, shape, dtype):
        return self.workspace.get(tag, shape, dtype)
