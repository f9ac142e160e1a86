"""Python handle on one ``stbpe_engine`` (one per GPU / rank)."""
from __future__ import annotations

import ctypes
import random
from typing import List, Optional, Sequence, Tuple

import numpy as np
import torch

from . import _lib as L


class CapacityError(RuntimeError):
    pass


def _raise(status: int, msg: str):
    if status == L.E_BADARG:
        raise ValueError(msg)
    if status == L.E_ID_OVERFLOW:
        raise OverflowError(msg)
    if status == L.E_CAPACITY:
        raise CapacityError(msg if "capacity exceeded" in msg else f"pair workspace capacity exceeded: {msg}")
    raise RuntimeError(msg)


def _stream_ptr(device: torch.device) -> ctypes.c_void_p:
    return ctypes.c_void_p(torch.cuda.current_stream(device).cuda_stream)


def trim_cache(device: Optional[torch.device | str | int] = None, keep_bytes: int = 0) -> None:
    """Give back the memory that destroyed engines left for the next one (at most 4 GiB per device, 64 MiB pinned), until
    at most ``keep_bytes`` of each stay; ``device`` None: of every device.  What ``torch.cuda.empty_cache`` is to torch's
    own cache, which cannot reach this one."""
    if device is None:
        indices = range(torch.cuda.device_count())
    else:
        index = torch.device("cuda", device).index if isinstance(device, int) else torch.device(device).index
        indices = [torch.cuda.current_device() if index is None else index]
    for i in (*indices, -1):
        st = L.load().stbpe_trim(i, int(keep_bytes))
        if st != L.OK:
            _raise(st, "bad device or size")


class Engine:
    """Token stream + pair table of one GPU.  Thin wrapper: every method is one C-ABI call."""

    def __init__(self, max_tokens: int, base_vocab: int = 256, max_merges: int = 50_000,
                 device: Optional[torch.device | str | int] = None, table_slots: int = 0,
                 world_size: int = 1, rank: int = 0):
        if not torch.cuda.is_available():
            raise RuntimeError("supertoken_b200 needs a CUDA device (B200, sm_100a); there is no CPU fallback")
        self._lib = L.load()
        dev = torch.device("cuda" if device is None else device)
        if dev.type != "cuda":
            raise ValueError("Engine runs on CUDA devices only")
        self.device = torch.device("cuda", torch.cuda.current_device() if dev.index is None else dev.index)
        self.base_vocab = int(base_vocab)
        self.max_merges = int(max_merges)
        self.world_size, self.rank = int(world_size), int(rank)
        cfg = L.Config(self.device.index, self.base_vocab, int(max_tokens), int(table_slots),
                       self.max_merges, self.world_size, self.rank, 0)
        self._h = ctypes.c_void_p()
        st = self._lib.stbpe_create(ctypes.byref(self._h), ctypes.byref(cfg))
        if st != L.OK:
            msg = self._lib.stbpe_last_error(None).decode()
            self._h = ctypes.c_void_p()
            _raise(st, msg)

    # ------------------------------------------------------------------ plumbing
    def _check(self, st: int):
        if st != L.OK:
            _raise(st, self._lib.stbpe_last_error(self._h).decode())

    def close(self):
        if getattr(self, "_h", None) and self._h.value:
            self._lib.stbpe_destroy(self._h)
            self._h = ctypes.c_void_p()

    def __del__(self):
        try:
            self.close()
        except Exception:
            pass

    @property
    def _s(self):
        return _stream_ptr(self.device)

    # ------------------------------------------------------------------ ingest
    def reset(self):
        self._check(self._lib.stbpe_reset(self._h))

    @staticmethod
    def _offsets(row_offsets, n: int) -> np.ndarray:
        if row_offsets is None:
            return np.array([0, n], dtype=np.int64)
        if isinstance(row_offsets, torch.Tensor):
            row_offsets = row_offsets.cpu().numpy()
        return np.ascontiguousarray(row_offsets, dtype=np.int64)

    def append_bytes(self, data, row_offsets=None):
        """``data``: uint8 torch tensor (CUDA or CPU, pinned or not) or numpy array."""
        if isinstance(data, np.ndarray):
            data = torch.from_numpy(np.ascontiguousarray(data, dtype=np.uint8))
        assert data.dtype == torch.uint8 and data.is_contiguous()
        off = self._offsets(row_offsets, data.numel())
        self._check(self._lib.stbpe_append_bytes(self._h, data.data_ptr(), data.numel(),
                                                 off.ctypes.data, len(off) - 1, self._s))

    def append_ids(self, ids, row_offsets=None):
        if isinstance(ids, np.ndarray):
            ids = torch.from_numpy(np.ascontiguousarray(ids, dtype=np.int32))
        assert ids.dtype == torch.int32 and ids.is_contiguous()
        off = self._offsets(row_offsets, ids.numel())
        self._check(self._lib.stbpe_append_ids(self._h, ids.data_ptr(), ids.numel(),
                                               off.ctypes.data, len(off) - 1, self._s))

    # ------------------------------------------------------------------ operators
    def count_initial(self):
        self._check(self._lib.stbpe_count_initial(self._h, self._s))

    def select_best(self, with_ties: bool = False) -> Tuple[Optional[int], int, int]:
        key, count, ties = ctypes.c_uint64(0), ctypes.c_int64(0), ctypes.c_int64(0)
        self._check(self._lib.stbpe_select_best(self._h, ctypes.byref(key), ctypes.byref(count),
                                                ctypes.byref(ties) if with_ties else None, self._s))
        if count.value <= 0:
            return None, 0, 0
        return int(key.value), int(count.value), int(ties.value)

    def apply_merge(self, a: int, b: int, new_id: int) -> int:
        if max(a, b, new_id) > 0x7FFFFFFE or min(a, b, new_id) < 0:
            raise OverflowError("Token id overflow: ids must be in [0, 2^31-2]")
        n = ctypes.c_int64(0)
        self._check(self._lib.stbpe_apply_merge(self._h, a, b, new_id, ctypes.byref(n), self._s))
        return int(n.value)

    def apply_merges(self, pairs: Sequence[Tuple[int, int]], first_new_id: int):
        """``apply_merge`` for every pair in order (new ids count up from ``first_new_id``), in one call."""
        if not pairs:
            return
        if max(max(a, b) for a, b in pairs) > 0x7FFFFFFE or min(min(a, b) for a, b in pairs) < 0 or \
                not 0 <= first_new_id <= 0x7FFFFFFE - (len(pairs) - 1):
            raise OverflowError("Token id overflow: ids must be in [0, 2^31-2]")
        p = np.asarray(pairs, dtype=np.int32)
        self._check(self._lib.stbpe_apply_merges(self._h, p.ctypes.data, len(p), int(first_new_id), self._s))

    def next_tied(self, merge: Optional[Tuple[int, int]] = None, new_id: int = 0, most: int = 0,
                  rng: Optional[random.Random] = None) -> Tuple[int, int, List[int]]:
        """One step of a loop that breaks ties: apply ``merge`` = (a, b) as ``new_id``, if given, go on
        with up to ``most`` best pairs while each is the only one with its count, and return the number of merges
        applied, the best count and the keys that hold it, ascending.  With ``rng`` ties are broken on the device too, as
        ``keys[rng.randrange(len(keys))]`` would, and ``rng`` is moved on by what that took; it may still return with a tie."""
        a, b = merge if merge is not None else (-1, -1)
        if max(a, b) > 0x7FFFFFFE or new_id + most > 0x7FFFFFFE or (merge is not None and min(a, b) < 0):
            raise OverflowError("Token id overflow: ids must be in [0, 2^31-2]")
        if getattr(self, "_tied", None) is None:
            self._tied, self._not_ahead, self._pause = np.empty(1024, dtype=np.uint64), 0, 0
        words, n_draws = None, 0
        # The generator's next outputs (the first one in the lowest bits), without moving it.  That costs some 15 us, so not
        # where the device breaks no tie: on 32-bit tokens (300 ties 26.3 ms, 22.2 without), and not for the next 1, 3, 7, 15,
        # 15, ... calls when it has left one to the host, as it does while more pairs are tied than it keeps or its list of
        # candidates is sure of (300 merges among 1 200 pairs: 2.2 of 83.8 ms).
        if rng is not None and most > 0 and self._not_ahead == 0 and self._lib.stbpe_token_bytes(self._h) == 2:
            n_draws = min(2 * most + 16, 1024)
            before = rng.getstate()
            words = rng.getrandbits(32 * n_draws).to_bytes(4 * n_draws, "little")
            rng.setstate(before)
        used = ctypes.c_int32(0)
        done, count, n = ctypes.c_int32(0), ctypes.c_int64(0), ctypes.c_int64(0)
        self._check(self._lib.stbpe_next_drawn(self._h, a, b, new_id, most, words, n_draws, ctypes.byref(used), ctypes.byref(done),
                                               ctypes.byref(count), self._tied.ctypes.data, len(self._tied), ctypes.byref(n),
                                               self._s))
        if used.value:
            rng.getrandbits(32 * used.value)
        if n_draws:
            self._pause = min(2 * self._pause + 1, 15) if not used.value and n.value > 1 else 0
            self._not_ahead = self._pause
        elif self._not_ahead:
            self._not_ahead -= 1
        if count.value <= 0:
            return done.value, 0, []
        if n.value > len(self._tied):
            return done.value, int(count.value), self.tied_keys(int(count.value), int(n.value))
        return done.value, int(count.value), self._tied[:n.value].tolist()

    def train(self, n_merges: int):
        self._check(self._lib.stbpe_train(self._h, int(n_merges), self._s))

    def train_timed(self, n_merges: int):
        """The merges of ``train`` one at a time; returns device milliseconds spent in (choices with the host's look at
        each, merges, 0, re-packs)."""
        ms = (ctypes.c_float * 4)()
        self._check(self._lib.stbpe_train_timed(self._h, int(n_merges), ms, self._s))
        return float(ms[0]), float(ms[1]), float(ms[2]), float(ms[3])

    def repack(self, force: bool = False) -> bool:
        """Dense re-pack of the stream if at most three quarters of the tile capacity are live (or forced)."""
        did = ctypes.c_int(0)
        self._check(self._lib.stbpe_repack(self._h, int(force), ctypes.byref(did), self._s))
        return bool(did.value)

    def count_error(self):
        """Raise the exception that matches the device error bits, if any are set."""
        st = self.state()
        bits = st.device_error
        if bits & 32:
            raise RuntimeError("a bounded device-side wait gave up (tile pipeline or a peer's flag)")
        if bits & (1 | 2 | 4):
            raise CapacityError("pair workspace capacity exceeded (pair table / delta buffers full)")
        if bits & 16:
            raise OverflowError("Token id overflow: ids must be in [0, 2^31-2]")
        if bits:
            raise RuntimeError(f"device error bits {bits:#x}")

    def state(self) -> L.State:
        st = L.State()
        self._check(self._lib.stbpe_get_state(self._h, ctypes.byref(st), self._s))
        return st

    def merges(self, first: int = 0, n: Optional[int] = None):
        """Returns (merges list[(a,b)], counts int64[n], live_before int64[n])."""
        if n is None:
            n = self.state().merges_done - first
        m = np.zeros((max(n, 0), 2), dtype=np.int32)
        c = np.zeros(max(n, 0), dtype=np.int64)
        lb = np.zeros(max(n, 0), dtype=np.int64)
        if n > 0:
            self._check(self._lib.stbpe_get_merges(self._h, first, n, m.ctypes.data, c.ctypes.data,
                                                   lb.ctypes.data))
        return list(zip(m[:, 0].tolist(), m[:, 1].tolist())), c, lb

    def export_histogram(self, cap: Optional[int] = None):
        """(keys int64 ascending, counts int64) on the device, zero counts dropped."""
        st = self.state()
        cap = int(cap if cap is not None else max(st.table_keys, 1))
        keys = torch.empty(cap, dtype=torch.int64, device=self.device)
        counts = torch.empty(cap, dtype=torch.int64, device=self.device)
        n = ctypes.c_int64(0)
        self._check(self._lib.stbpe_export_histogram(self._h, keys.data_ptr(), counts.data_ptr(), cap,
                                                     ctypes.byref(n), self._s))
        return keys[:n.value], counts[:n.value]

    def tied_keys(self, count: int, n_ties: int) -> List[int]:
        """Keys holding exactly ``count``, ascending."""
        buf = torch.empty(max(n_ties, 1), dtype=torch.int64, device=self.device)
        n = ctypes.c_int64(0)
        self._check(self._lib.stbpe_export_ties(self._h, count, buf.data_ptr(), buf.numel(),
                                                ctypes.byref(n), self._s))
        return sorted(int(k) for k in buf[:min(n.value, buf.numel())].cpu().numpy().view(np.uint64))

    def export_stream(self):
        """int32 ids on the device with bit 31 marking row starts -> (ids, row_offsets) on CPU."""
        st = self.state()
        cap = max(int(st.live_tokens), 1)
        buf = torch.empty(cap, dtype=torch.int32, device=self.device)
        n = ctypes.c_int64(0)
        self._check(self._lib.stbpe_export_stream(self._h, buf.data_ptr(), cap, ctypes.byref(n), self._s))
        raw = buf[:n.value].cpu().numpy().view(np.uint32)
        starts = np.nonzero(raw >> 31)[0].astype(np.int64)
        ids = (raw & 0x7FFFFFFF).astype(np.int32)
        off = np.concatenate([starts, [len(ids)]]).astype(np.int64) if len(ids) else np.zeros(1, np.int64)
        return ids, off
