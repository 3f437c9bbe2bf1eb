"""GPU-side construction of the wire format the operators consume (`unique_slots`, `pad_mask`, `c_base`) from
per-document slot state that stays resident on the GPU.

The reference builds these per chunk on the host: `WikiTextMMapDataset.__getitem__` (mathbrain/data.py:95-148) looks
the document's history up in Python loops and reads `states.bin`, and `dynamic_collate_fn` (mathbrain/data.py:211-235)
pads and stacks.  Here a `ChunkFeeder` holds, for B documents in flight, the state of every slot after its last update
and the step of that update (the layout of `DecodeState`), and for the next chunk of every document

    batch = feeder.next_batch(x, fill)        # x [B, T] int64 on the GPU, fill [B] valid lengths
    ...   C_seq = compute_query_ema_history(x, rhos, V, batch["c_base"], batch["unique_slots"]); the model step ...
    feeder.advance(x, fill, C_seq)            # the documents move on by `fill` tokens

builds `unique_slots` (the chunk's sorted distinct tokens first, then the sorted history-only tokens: the order of
mathbrain/data.py:104-124), `pad_mask` and `c_base` (state decayed to the chunk's first step, mathbrain/data.py:128-140)
with two kernels (csrc/feed.cu); the only host synchronisation is the read of the widest slot list, which the
reference's model does as well (mathbrain/model.py:169).
"""
import torch

from . import _lib
from .ops import _ptr, _require_cuda, _stream


class ChunkFeeder:
    def __init__(self, n_docs, vocab, rhos, capacity=8192, device="cuda"):
        _require_cuda(rhos)
        dev = torch.device(device) if device is not None else rhos.device
        self.B, self.V, self.N, self.cap = int(n_docs), int(vocab), int(rhos.shape[0]), int(capacity)
        self.rhos = rhos.float().contiguous().to(dev)
        self.state = torch.zeros(self.B, self.V, self.N, dtype=torch.float32, device=dev)   # value after the last update
        self.last_t = torch.full((self.B, self.V), -1, dtype=torch.int32, device=dev)        # step of that update
        self.seen = torch.zeros(self.B, self.cap, dtype=torch.int64, device=dev)             # tokens seen so far, per document
        self.n_seen = torch.zeros(self.B, dtype=torch.int64, device=dev)
        self.t0 = torch.zeros(self.B, dtype=torch.int32, device=dev)                         # step of the next chunk's first token
        self._widest = None        # (widest slot list, the seen lists it was read from) of a next_batch that no advance has followed yet

    def reset(self, docs):
        """Start new documents in the given rows (a tensor or list of row numbers)."""
        docs = torch.as_tensor(docs, dtype=torch.long, device=self.state.device)
        self.state[docs] = 0
        self.last_t[docs] = -1
        self.n_seen[docs] = 0
        self.t0[docs] = 0

    def _same_device(self, *operands):
        """Every tensor whose address goes to a kernel, the resident ones included (a program may have put others in their
        place), is on the state's device; resident ones of another type or layout are brought into the kernels'."""
        dev = self.state.device
        for t in operands:
            if t.device != dev:
                raise _lib.MbemaError("ChunkFeeder: operand on %s, state on %s" % (t.device, dev))
        B, V, N, cap = self.B, self.V, self.N, self.cap
        for name, dtype, shape in (("state", torch.float32, (B, V, N)), ("last_t", torch.int32, (B, V)), ("seen", torch.int64, (B, cap)),
                                   ("n_seen", torch.int64, (B,)), ("t0", torch.int32, (B,)), ("rhos", torch.float32, (N,))):
            t = getattr(self, name)
            if t.device != dev or t.shape != shape:
                raise _lib.MbemaError("ChunkFeeder: %s is %s on %s, expected %s on %s" % (name, tuple(t.shape), t.device, shape, dev))
            if t.dtype != dtype or not t.is_contiguous():
                setattr(self, name, t.to(dtype).contiguous())

    def _lists(self):
        """The seen lists as they stand: the tensors with their version counters, which in-place changes raise (tensors made
        under inference_mode have none)."""
        return [(t, None if t.is_inference() else t._version) for t in (self.seen, self.n_seen)]

    def _longest_possible(self, T):
        """No seen list is longer after a chunk of T tokens: the lists of the next_batch just before hold every token seen so
        far, unless the program has changed them since."""
        widest, self._widest = self._widest, None
        if widest is None or any(a is not b or v is None or v != w for (a, v), (b, w) in zip(widest[1], self._lists())):
            return self.cap + 1
        return min(widest[0] + T, self.V)

    def next_batch(self, x, fill):
        """Wire format of the next chunk of every document: dict(unique_slots [B, K] int64 (0-padded, as the collate
        function pads), pad_mask [B, K] bool, c_base [B, K, N] float32, K_max).  x [B, T] int64, fill [B] valid lengths."""
        _require_cuda(x, fill)
        self._same_device(x, fill)
        with torch.cuda.device(self.state.device):
            return self._next_batch(x, fill)

    def _chunk(self, x, fill):
        if x.dim() != 2 or x.shape[0] != self.B:
            raise _lib.MbemaError("ChunkFeeder: chunk of shape %s for %d documents" % (tuple(x.shape), self.B))
        return x.long().contiguous(), fill.to(torch.int32).expand(self.B).contiguous()

    def _next_batch(self, x, fill):
        B, T = x.shape
        dev = x.device
        lib = _lib.load()
        x, fill = self._chunk(x, fill)
        lists = torch.empty(B, T + self.cap, dtype=torch.int32, device=dev)
        counts = torch.empty(B + 1, dtype=torch.int32, device=dev)
        rc = lib.mbema_feed_lists(_ptr(x), _ptr(fill), _ptr(self.seen), _ptr(self.n_seen), _ptr(lists), _ptr(counts), B, T, self.V,
                                  self.cap, _stream())
        _lib.check(rc, "mbema_feed_lists")
        widest = int(counts[B])                                                  # the one host synchronisation
        self._widest = widest, self._lists()
        K = max(16, widest)
        unique = torch.empty(B, K, dtype=torch.int64, device=dev)
        pad_mask = torch.empty(B, K, dtype=torch.bool, device=dev)
        c_base = torch.empty(B, K, self.N, dtype=torch.float32, device=dev)
        rc = lib.mbema_feed_batch(_ptr(lists), _ptr(counts), _ptr(self.state), _ptr(self.last_t), _ptr(self.t0), _ptr(self.rhos),
                                  _ptr(unique), _ptr(pad_mask), _ptr(c_base), B, K, T, self.V, self.N, self.cap, _stream())
        _lib.check(rc, "mbema_feed_batch")
        return dict(unique_slots=unique, pad_mask=pad_mask, c_base=c_base, K_max=K)

    def advance(self, x, fill, C_seq):
        """Move every document past its chunk: the state of each token of the chunk becomes the query-side state at its
        LAST occurrence plus one (C_seq from compute_query_ema_history on this chunk), stamped with that step; tokens seen
        for the first time join the document's list.  Raises if a list would overflow."""
        _require_cuda(x, fill, C_seq)
        self._same_device(x, fill, C_seq)
        with torch.cuda.device(self.state.device):
            self._advance(x, fill, C_seq)

    def _advance(self, x, fill, C_seq):
        B, T = x.shape
        x, fill = self._chunk(x, fill)
        C_seq = C_seq[:B, :T].float().contiguous()
        if C_seq.shape != (B, T, self.N):
            raise _lib.MbemaError("ChunkFeeder: C_seq must be [%d, %d, %d]" % (B, T, self.N))

        def call(status, check):
            rc = _lib.load().mbema_feed_advance(_ptr(x), _ptr(fill), _ptr(C_seq), _ptr(self.state), _ptr(self.last_t), _ptr(self.seen),
                                                _ptr(self.n_seen), _ptr(self.t0), _ptr(status), B, T, self.V, self.N, self.cap, check,
                                                _stream())
            _lib.check(rc, "mbema_feed_advance")

        # Where an overflow is ruled out nothing is asked of the device (a read back costs as much as the three kernels).
        if self._longest_possible(T) > self.cap:
            status = torch.zeros(1, dtype=torch.int32, device=x.device)
            call(status, 1)
            if int(status) > self.cap:
                raise _lib.MbemaError("ChunkFeeder: the list of seen tokens is full (capacity %d)" % self.cap)
        call(None, 0)
