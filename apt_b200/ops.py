"""Host side of the data path: the operators of the reference's ``npc`` library
(``TORCH_LIBRARY(npc, m)``, src/pybind.cc:18-48) with the same names, argument
meaning and result layout, implemented on libapt_b200's C ABI.

PyTorch is used for device memory, streams and ``torch.distributed`` only; all
arithmetic of the path runs in the CUDA library. There is no CPU fallback:
every operator except ``cpu_load_subtensor`` requires CUDA tensors.

State lives in one process-wide object like the reference's ``NPCState``
(src/state.h:32-63): one process drives one GPU.
"""
import contextlib
import ctypes
import os
import threading
from typing import List, Optional, Tuple

import torch

from . import _lib, _native
from ._lib import check, lib

_DTYPE_CODE = {torch.float32: _lib.F32, torch.bfloat16: _lib.BF16, torch.float16: _lib.F16}


def _ptr(t: Optional[torch.Tensor]):
    if t is None or t.numel() == 0:
        return None
    return ctypes.c_void_p(t.data_ptr())


def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def _need_cuda(t: torch.Tensor, name: str, dtype=torch.int64):
    if not t.is_cuda:
        raise RuntimeError(f"{name} must be a CUDA tensor (apt_b200 has no CPU path)")
    if dtype is not None and t.dtype != dtype:
        raise RuntimeError(f"{name} must have dtype {dtype}, got {t.dtype}")
    return t.contiguous()


def _device_visible(t: torch.Tensor, name: str) -> torch.Tensor:
    """A tensor kernels can dereference: CUDA memory, or page-locked host memory
    (registered here if needed, as the reference's pin_tensor does,
    python/npc/utils/utils.py:70-75)."""
    if t.is_cuda:
        return t.contiguous()
    if not t.is_contiguous():
        raise RuntimeError(f"{name} must be contiguous")
    if t.numel() > 0 and not t.is_pinned():
        from . import hostmem

        hostmem.register(t.data_ptr(), t.numel() * t.element_size())
    return t


class FeatStorage:
    """FeatStorage, src/state.h:10-16."""

    def __init__(self):
        self.dev_feats = None
        self.uva_feats = None
        self.feat_pos_map = None
        self._cpu_feat_pos_map = None
        self._cpu_map_args = None
        self.num_total_nodes = 0
        self.feat_dim = 0
        self.rank_feat_dim = 0
        self.feat_dim_offset = 0

    @property
    def cpu_feat_pos_map(self):
        if self._cpu_feat_pos_map is None and self._cpu_map_args is not None:
            n, localnode_idx = self._cpu_map_args
            m = torch.full((n,), -1, dtype=torch.int64)
            m[localnode_idx] = -torch.arange(localnode_idx.numel(), dtype=torch.int64) - 2
            self._cpu_feat_pos_map = m
        return self._cpu_feat_pos_map


class GraphStorage:
    """GraphStorage, src/state.h:18-23."""

    def __init__(self):
        self.dev_indptr = None
        self.dev_indices = None
        self.uva_indptr = None
        self.uva_indices = None
        self.adj_pos_map = None
        self.num_total_nodes = 0
        self.num_cached_nodes = 0


class NPCState:
    """NPCState, src/state.h:32-63, plus what the CUDA library needs from the
    host: cached workspaces, the device status word and the exchange backend."""

    def __init__(self):
        self.rank = 0
        self.local_rank = 0
        self.world_size = 1
        self.node_size = 1
        self.initialized = False
        self.shuffle_min_vids = None
        self._min_vids_host = None
        self.shuffle_id_offset = 0
        self.graph = GraphStorage()
        self.feat = FeatStorage()
        self.sample_key = 7777777  # the reference's seed constant, src/cuda/npc_kernel.cu:292
        self.sample_calls = 0
        self.sample_replace = True
        self._ws = {}
        self._lane_words = {}
        # mini-batches that run beside one another on the GPU (each on a stream of its own) must not
        # share scratch: workspaces, the word block and the exchange context are kept per lane
        self._tls = threading.local()
        self._lane_exchange = {}
        self._lane_streams = {}
        self.prefetched = None  # _RowsAhead a sampler left for the next load_subtensor
        self._publish_seq = 0
        self._seq_lock = threading.Lock()
        self.generation = 0     # bumped whenever installed state changes; captured graphs check it
        self.profiling = False
        self.exchange = None  # set by apt_b200.exchange.make_exchange at init
        self.exchange_generation = 0
        self._side_streams = {}
        self.shuffle_backend = os.environ.get("APT_SHUFFLE_BACKEND", "p2p")
        self.p2p_region_bytes = int(os.environ.get("APT_P2P_REGION_MB", "256")) << 20
        # inboxes of the lanes beside the first carry the samplers' id exchanges only
        self.p2p_lane_region_bytes = int(os.environ.get("APT_P2P_LANE_REGION_MB", "64")) << 20

    @property
    def lane(self) -> int:
        """The lane whose scratch the calling thread's operators use (0: the caller's own)."""
        return getattr(self._tls, "lane", 0)

    @lane.setter
    def lane(self, value: int):
        self._tls.lane = int(value)

    # -- device scratch --------------------------------------------------
    def device(self):
        return torch.device("cuda", torch.cuda.current_device())

    def workspace(self, name: str, nbytes: int) -> torch.Tensor:
        """A cached, 256-byte aligned scratch tensor of at least nbytes."""
        key = (name, torch.cuda.current_device(), self.lane)
        buf = self._ws.get(key)
        if buf is None or buf.numel() < nbytes:
            buf = torch.empty(max(int(nbytes * 1.25), 1 << 16), dtype=torch.uint8, device=self.device())
            self._ws[key] = buf
        return buf

    def side_stream(self, k: int = 0) -> torch.cuda.Stream:
        """Further streams of this device for work that runs beside the main chain of a mini-batch."""
        key = (k, torch.cuda.current_device())
        stream = self._side_streams.get(key)
        if stream is None:
            stream = self._side_streams[key] = torch.cuda.Stream(device=self.device())
        return stream

    @contextlib.contextmanager
    def beside(self, k: int):
        """Enqueues the block's work on side stream k, behind what the current stream holds so far. The current stream
        waits for it with `join(k)`."""
        side = self.side_stream(k)
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            yield

    def join(self, k: int):
        torch.cuda.current_stream().wait_stream(self.side_stream(k))

    @contextlib.contextmanager
    def joined_if_it_fails(self, *sides: Optional[int]):
        """For what runs while side streams are at work (None: no such stream). Where it raises, the current stream waits for them all the
        same: their buffers are given back and their scratch is the next caller's."""
        try:
            yield
        except BaseException:
            for k in sides:
                if k is not None:
                    self.join(k)
            raise

    def lane_stream(self, lane: int) -> torch.cuda.Stream:
        """The one stream on which work that uses lane `lane`'s scratch is enqueued: everything on
        a lane runs in order, whichever sampler put it there."""
        key = (lane, torch.cuda.current_device())
        stream = self._lane_streams.get(key)
        if stream is None:
            stream = self._lane_streams[key] = torch.cuda.Stream(device=self.device())
        return stream

    NUM_WORDS = 256

    def words(self) -> torch.Tensor:
        """int64[256] device words: [0..254] small results (counts a kernel leaves for
        the next kernel and, later, for the host), [255] status flags. Inside own_words() the small results are in
        a block of the caller's."""
        tls = self._tls
        own = getattr(tls, "words", None)
        if own is not None:
            return own
        words = self._lane_words.get(getattr(tls, "lane", 0))
        return words if words is not None and words.get_device() == torch.cuda.current_device() else self.lane_words()

    @contextlib.contextmanager
    def own_words(self, words: torch.Tensor):
        """Small results of the block's operators go to `words`; status flags stay in the lane's block. For operators that
        are still reading their counts when others have begun to write theirs."""
        self._tls.words = words
        try:
            yield
        finally:
            self._tls.words = None

    def lane_words(self) -> torch.Tensor:
        """The word block of the calling thread's lane, its status flags among them."""
        words = self._lane_words.get(self.lane)
        if words is None or words.device != self.device():
            words = self._lane_words[self.lane] = torch.zeros(self.NUM_WORDS, dtype=torch.int64, device=self.device())
        return words

    def host_words(self) -> torch.Tensor:
        """The calling thread's page-locked copy of a word block, with a sequence number in its words. Threads that read at the
        same time have one each: a reader polls its copy for its own number."""
        host = getattr(self._tls, "host", None)
        if host is None:
            host = self._tls.host = _native.pinned_words(self.NUM_WORDS)
        return host

    def word(self, k: int) -> torch.Tensor:
        """One-element view of device word k (a device-side count)."""
        return self.words()[k:k + 1]

    def status_ptr(self):
        return ctypes.c_void_p(self.lane_words().data_ptr() + 8 * (self.NUM_WORDS - 1))

    def read_words(self) -> torch.Tensor:
        """Copies the device words to the host (one stream sync) and raises on
        any status flag except zero-degree, which is only a notice."""
        status, host = self.lane_words(), self.host_words()
        self.check_flags(_native.read_words(self.words(), status, host, self.next_sequence()))
        return host

    def next_sequence(self) -> int:
        """A number no earlier publication of a word block carries."""
        with self._seq_lock:
            self._publish_seq += 1
            return self._publish_seq

    def check_host_words(self, host: torch.Tensor):
        """Raises if a host copy of the word block carries a status flag (zero-degree is a notice)."""
        self.check_flags(int(host[self.NUM_WORDS - 1]) & 0xFFFFFFFF)

    def check_flags(self, flags: int):
        if flags & ~_lib.FLAG_ZERO_DEGREE:
            self.lane_words()[self.NUM_WORDS - 1] = 0
            raise RuntimeError(f"apt_b200 device status flags 0x{flags:x}: " + _flag_text(flags))


def _flag_text(flags):
    names = {
        _lib.FLAG_ID_OUT_OF_RANGE: "id outside the registered tables",
        _lib.FLAG_FEAT_NOT_EXIST: "feature row neither cached nor in host memory",
        _lib.FLAG_ZERO_DEGREE: "node without in-neighbours sampled",
        _lib.FLAG_TABLE_FULL: "workspace or inbox region too small",
        _lib.FLAG_PEER_TIMEOUT: "a peer's data did not arrive within the wait bound (APT_P2P_TIMEOUT_MS); the "
                                "exchange refuses further use: call init() again on every rank, behind a barrier",
        _lib.FLAG_NOT_GROUPED: "edges of a block are not grouped by destination",
        _lib.FLAG_SIZE_MISMATCH: "a peer sent another number of rows than the reduction expects",
        _lib.FLAG_COPY_TIMEOUT: "input rows of a sum did not reach shared memory in time; some of its rows are zero",
    }
    return ", ".join(v for k, v in names.items() if flags & k)


STATE = NPCState()


def _version(t: torch.Tensor):
    """PyTorch's count of the in-place changes of a tensor (inference tensors keep none)."""
    return None if t.is_inference() else t._version


def _tables_key():
    """What a gather's rows depend on beside their ids: a gather enqueued under one key is good for as long as the key is the
    same. Covers another feature table being installed and changes of an installed one that PyTorch knows of."""
    f = STATE.feat
    return STATE.generation, _version(f.dev_feats), _version(f.uva_feats)


class _RowsAhead:
    """Feature rows that a sampler gathered for `ids`, its input nodes, under `key`. `pending` (None: nothing to wait for)
    orders a stream behind the gather."""

    def __init__(self, ids, rows, key, pending):
        self.ids, self.rows, self.key, self.pending = ids, rows, key, pending
        self.version = _version(ids)

    def serves(self, node_id) -> bool:
        ids = self.ids
        if self.key != _tables_key() or self.version != _version(ids):
            return False
        return ids is node_id or (ids.data_ptr() == node_id.data_ptr() and ids.numel() == node_id.numel()
                                  and ids.dtype == node_id.dtype and node_id.is_contiguous())



def _exchange():
    """The exchange backend; a process that never called init() is a world of one. Lanes other
    than the first get a context of their own on first use (a collective step: every rank has to
    reach it, which holds when the ranks run the same sampler), since the flags of one context
    order its exchanges as one sequence."""
    if STATE.exchange is None:
        from .exchange import make_exchange

        STATE.exchange = make_exchange(STATE)
    if STATE.lane == 0 or STATE.exchange.name != "p2p" or STATE.world_size == 1:
        return STATE.exchange
    ex = STATE._lane_exchange.get(STATE.lane)
    if ex is None or ex.generation != STATE.exchange_generation:
        from .exchange import P2PExchange

        ex = P2PExchange(STATE, min(STATE.p2p_region_bytes, STATE.p2p_lane_region_bytes))
        ex.generation = STATE.exchange_generation
        STATE._lane_exchange[STATE.lane] = ex
    return ex


def profile_enable(on: bool):
    """Per-kernel CUDA-event timing (apt_profile_enable). Captured CUDA graphs
    cannot hold timing events, so samplers run eagerly while this is on."""
    STATE.profiling = bool(on)
    check(lib.apt_profile_enable(1 if on else 0))


def check_status():
    """Synchronises and raises if any kernel since the last check flagged an error."""
    STATE.read_words()


# ---------------------------------------------------------------- init / state
def nccl_get_unique_id() -> torch.Tensor:
    """NCCLGetUniqueId, src/core.cc:38-44: int64[16] on the CPU. The exchange
    here rides on torch.distributed's process group, so the id is a
    placeholder kept for callers that broadcast it (python/npc/__init__.py:33-49)."""
    return torch.zeros(16, dtype=torch.int64)


def init(rank: int, local_rank: int, world_size: int, nccl_id_tensor_list: torch.Tensor, node_size: int) -> None:
    """Initialize, src/core.cc:54-100."""
    from .exchange import make_exchange

    s = STATE
    s.rank, s.local_rank, s.world_size, s.node_size = int(rank), int(local_rank), int(world_size), int(node_size)
    torch.cuda.set_device(s.local_rank)
    s.exchange = make_exchange(s)
    s.exchange_generation += 1
    for ex in s._lane_exchange.values():
        ex.close()
    s._lane_exchange = {}
    s.initialized = True
    s.generation += 1


def register_min_vids(shuffle_min_vids: torch.Tensor, shuffle_id_offset: int = 0) -> None:
    """RegisterMinVids, src/core.cc:102-108."""
    mv = shuffle_min_vids.to(device=STATE.device(), dtype=torch.int64).contiguous()
    if mv.numel() != STATE.world_size + 1:
        raise RuntimeError(f"min_vids needs world_size+1 = {STATE.world_size + 1} entries, got {mv.numel()}")
    STATE.shuffle_min_vids = mv
    STATE.generation += 1
    STATE._min_vids_host = [int(x) for x in shuffle_min_vids.cpu().tolist()]
    STATE.shuffle_id_offset = int(shuffle_id_offset)


def mix_cache_graphs(num_cached_nodes: int, cached_node_idx: torch.Tensor, cached_indptr: torch.Tensor,
                     cached_indices: torch.Tensor, global_indptr: torch.Tensor, global_indices: torch.Tensor) -> None:
    """MixCacheGraphs, src/cache_graphs.cc:12-49. The global CSC may be pinned
    host memory (read over the host link, as in the reference) or CUDA memory
    (the whole topology resident in HBM)."""
    g = STATE.graph
    STATE.generation += 1
    if int(num_cached_nodes) != cached_node_idx.numel():
        raise RuntimeError("num_cached_nodes != cached_node_idx.numel()")
    g.num_cached_nodes = int(num_cached_nodes)
    g.num_total_nodes = global_indptr.numel() - 1
    g.uva_indptr = _device_visible(global_indptr, "global_indptr")
    g.uva_indices = _device_visible(global_indices, "global_indices")
    if g.num_cached_nodes > 0:
        g.dev_indptr = _need_cuda(cached_indptr, "cached_indptr")
        g.dev_indices = _need_cuda(cached_indices, "cached_indices")
        m = -torch.arange(g.num_total_nodes, dtype=torch.int64, device=STATE.device()) - 2
        m[cached_node_idx.to(STATE.device())] = torch.arange(g.num_cached_nodes, dtype=torch.int64, device=STATE.device())
        g.adj_pos_map = m
    else:
        # Every node reads the global CSC: the position map would be the
        # identity encoding, so it is not materialised.
        g.dev_indptr = g.dev_indices = g.adj_pos_map = None


def cache_feats_shared(num_total_nodes: int, localnode_feats: torch.Tensor, cached_feats: torch.Tensor,
                       cached_idx: torch.Tensor, localnode_idx: torch.Tensor, feat_dim_offset: int = 0) -> None:
    """CacheFeatsShared, src/cache_feats.cc:14-61."""
    f = STATE.feat
    dev = STATE.device()
    STATE.generation += 1
    if localnode_feats.dim() != 2 or cached_feats.dim() != 2:
        raise RuntimeError("feature tables must be 2-D")
    if cached_feats.dtype != localnode_feats.dtype or cached_feats.dtype not in _DTYPE_CODE:
        raise RuntimeError(f"unsupported feature dtypes {localnode_feats.dtype}/{cached_feats.dtype}")
    f.num_total_nodes = int(num_total_nodes)
    f.uva_feats = _device_visible(localnode_feats, "localnode_feats")
    f.dev_feats = _need_cuda(cached_feats, "cached_feats", dtype=None)
    f.feat_dim = localnode_feats.shape[1]
    f.rank_feat_dim = cached_feats.shape[1]
    f.feat_dim_offset = int(feat_dim_offset)
    m = torch.full((f.num_total_nodes,), -1, dtype=torch.int64, device=dev)
    li = localnode_idx.to(dev)
    m[li] = -torch.arange(li.numel(), dtype=torch.int64, device=dev) - 2
    m[cached_idx.to(dev)] = torch.arange(cached_idx.numel(), dtype=torch.int64, device=dev)
    f.feat_pos_map = m
    f._cpu_feat_pos_map = None
    f._cpu_map_args = (f.num_total_nodes, localnode_idx.cpu())


def set_sampling(key: Optional[int] = None, call_id: Optional[int] = None, replace: Optional[bool] = None):
    """Sampler stream control: draws depend only on (key, call_id, seed slot,
    draw slot); call_id advances by one per sampling call. Captured mini-batches carry the key and the mode, not the
    call id: they stay as they are when only that changes."""
    if (key is not None and int(key) != STATE.sample_key) or (replace is not None and bool(replace) != STATE.sample_replace):
        STATE.generation += 1
    if key is not None:
        STATE.sample_key = int(key)
    if call_id is not None:
        STATE.sample_calls = int(call_id)
    if replace is not None:
        STATE.sample_replace = bool(replace)


# -------------------------------------------------------------------- sampling
def _sample(seeds: torch.Tensor, fanout: int, n_dev: Optional[torch.Tensor] = None,
            call_id: Optional[int] = None, call_base_dev: Optional[torch.Tensor] = None) -> torch.Tensor:
    """n_dev: optional one-element device count; seeds.numel() is then an upper bound.
    call_id / call_base_dev: explicit call id (plus a device-side base) instead of the
    process-wide counter, for sequences replayed from a CUDA graph."""
    g = STATE.graph
    if g.uva_indptr is None:
        raise RuntimeError("mix_cache_graphs has not been called")
    seeds = _need_cuda(seeds, "seeds")
    out = torch.empty(seeds.numel() * int(fanout), dtype=torch.int64, device=seeds.device)
    if call_id is None:
        call_id = STATE.sample_calls
        STATE.sample_calls += 1
    check(lib.apt_sample_csc_fanout(
        _ptr(seeds), seeds.numel(), _ptr(n_dev), int(fanout), _ptr(g.adj_pos_map), g.num_total_nodes,
        _ptr(g.dev_indptr), _ptr(g.dev_indices), _ptr(g.uva_indptr), _ptr(g.uva_indices),
        STATE.sample_key, call_id & 0xFFFFFFFF, _ptr(call_base_dev), 1 if STATE.sample_replace else 0,
        _ptr(out), STATE.status_ptr(), _stream()))
    return out


def local_sample_one_layer(seeds: torch.Tensor, fanout: int) -> List[torch.Tensor]:
    """LocalSamplingNeibhorsOneLayer, src/sampling.cc:13-17: [seeds, neighbors]."""
    return [seeds, _sample(seeds, fanout)]


def _relabel_enqueue(seeds, neighbors, n_dev, count_out):
    """Enqueues the relabelling; the number of unique ids lands in the device
    word `count_out`. Returns the full-length (upper bound) buffers."""
    n = seeds.numel() + neighbors.numel()
    uniq = torch.empty(n, dtype=torch.int64, device=seeds.device)
    rel = torch.empty(neighbors.numel(), dtype=torch.int64, device=seeds.device)
    ws = _relabel_workspace(n)
    check(lib.apt_relabel_csc(_ptr(seeds), seeds.numel(), _ptr(n_dev), _ptr(neighbors), neighbors.numel(),
                              _ptr(ws), ws.numel(), _ptr(uniq), _ptr(rel),
                              _ptr(count_out), STATE.status_ptr(), _stream()))
    return uniq, rel


def _relabel_workspace(n):
    ws = STATE.workspace("relabel", lib.apt_relabel_workspace_bytes(n))
    if getattr(ws, "_apt_clean", False) is not True:
        # the table has to be empty once; every call then releases the slots it used
        check(lib.apt_relabel_workspace_init(_ptr(ws), ws.numel(), _stream()))
        ws._apt_clean = True
    return ws


def _row_tables():
    """(position map, nodes, cached rows, host rows) for the kernels that look ids of a gather up."""
    f = STATE.feat
    if f.feat_pos_map is None:
        return None, 0, 0, 0
    return _ptr(f.feat_pos_map), f.num_total_nodes, f.dev_feats.shape[0], f.uva_feats.shape[0]


def _sample_relabel_enqueue(seeds, fanout, n_dev, count_out, call_id=None, call_base_dev=None, want_neighbors=False,
                            look_up=False):
    """One sampled layer, sampling and relabelling together (apt_sample_relabel_block): returns the
    upper-bound buffers (unique ids, relabelled neighbours, neighbours or None); the number of
    unique ids lands in the device word `count_out`. `look_up`: the unique ids are those of a gather,
    flag what it would flag."""
    g = STATE.graph
    if g.uva_indptr is None:
        raise RuntimeError("mix_cache_graphs has not been called")
    if not STATE.sample_replace:
        nbr = _sample(seeds, fanout, n_dev, call_id, call_base_dev)
        uniq, rel = _relabel_enqueue(seeds, nbr, n_dev, count_out)
        if look_up:
            none = torch.empty(0, dtype=torch.int64, device=uniq.device)
            concat_ids(none, None, uniq, count_out, None, look_up=True)
        return uniq, rel, nbr
    seeds = _need_cuda(seeds, "seeds")
    S, f = seeds.numel(), int(fanout)
    uniq = torch.empty(S * (1 + f), dtype=torch.int64, device=seeds.device)
    rel = torch.empty(S * f, dtype=torch.int64, device=seeds.device)
    nbr = torch.empty(S * f, dtype=torch.int64, device=seeds.device) if want_neighbors else None
    ws = _relabel_workspace(S * (1 + f))
    if call_id is None:
        call_id = STATE.sample_calls
        STATE.sample_calls += 1
    check(lib.apt_sample_relabel_block(
        _ptr(seeds), S, _ptr(n_dev), f, _ptr(g.adj_pos_map), g.num_total_nodes, _ptr(g.dev_indptr),
        _ptr(g.dev_indices), _ptr(g.uva_indptr), _ptr(g.uva_indices), STATE.sample_key, call_id & 0xFFFFFFFF,
        _ptr(call_base_dev), _ptr(ws), ws.numel(), _ptr(nbr), _ptr(uniq), _ptr(rel), None, _ptr(count_out),
        *(_row_tables() if look_up else (None, 0, 0, 0)), STATE.status_ptr(), _stream()))
    return uniq, rel, nbr


def relabel_csc(seeds: torch.Tensor, neighbors: torch.Tensor) -> List[torch.Tensor]:
    """RelabelCSC, src/relabel.cc:9-15: [all_unique, relabeled_neighbors]."""
    seeds = _need_cuda(seeds, "seeds")
    neighbors = _need_cuda(neighbors, "neighbors")
    uniq, rel = _relabel_enqueue(seeds, neighbors, None, STATE.word(0))
    num_unique = int(STATE.read_words()[0])
    return [uniq[:num_unique], rel]


# ---------------------------------------------------------------- seed shuffle
def _bucket(seeds: torch.Tensor, n_dev: Optional[torch.Tensor] = None, sizes: Optional[torch.Tensor] = None,
            offsets: Optional[torch.Tensor] = None):
    """Stable partition by owner: (sorted ids, permutation, sizes[world_size + 1]
    with their total last, inclusive offsets[world_size]). `sizes` / `offsets`
    may be given as preallocated device views."""
    s = STATE
    if s.shuffle_min_vids is None:
        raise RuntimeError("register_min_vids has not been called")
    n = seeds.numel()
    dev = seeds.device
    sorted_ids = torch.empty(n, dtype=torch.int64, device=dev)
    perm = torch.empty(n, dtype=torch.int64, device=dev)
    if sizes is None:
        sizes = torch.empty(s.world_size + 1, dtype=torch.int64, device=dev)
    if offsets is None:
        offsets = torch.empty(s.world_size, dtype=torch.int64, device=dev)
    nbytes = lib.apt_bucket_workspace_bytes(n, s.world_size)
    ws = s.workspace("bucket", nbytes)
    node_beg = s.rank - s.rank % s.node_size
    check(lib.apt_bucket_by_owner(_ptr(seeds), n, _ptr(n_dev), _ptr(s.shuffle_min_vids), s.world_size,
                                  s.shuffle_id_offset,
                                  s.rank, node_beg, node_beg + s.node_size, _ptr(ws), ws.numel(),
                                  _ptr(sorted_ids), _ptr(perm), _ptr(sizes), _ptr(offsets), _stream()))
    return sorted_ids, perm, sizes, offsets


def shuffle_seeds(seeds: torch.Tensor) -> Tuple[torch.Tensor, torch.Tensor, torch.Tensor, torch.Tensor]:
    """ShuffleSeeds, src/sampling.cc:159-193: (recv_frontier [cuda],
    permutation [cuda], recv_offset [cpu], dev_offset [cpu]); offsets are
    inclusive cumulative counts. Ids of one owner keep their input order."""
    seeds = _need_cuda(seeds, "seeds")
    sorted_ids, perm, sizes, offsets = _bucket(seeds)
    recv, recv_offset, dev_offset = _exchange().exchange_ids(sorted_ids, sizes, offsets)
    return recv, perm, recv_offset, dev_offset


def unique_sorted(ids: torch.Tensor, id_lo: int, id_hi: int):
    """Sorted unique + inverse of ids in [id_lo, id_hi): torch::_unique2(sorted,
    return_inverse) of src/sampling.cc:58-59, via a bitmap over the id range."""
    ids = _need_cuda(ids, "ids")
    uniq, inv = _unique_enqueue(ids, None, id_lo, id_hi, STATE.word(0))
    num_unique = int(STATE.read_words()[0])
    return uniq[:num_unique], inv


def _unique_bitmap(rng, ws_name):
    """The cached bitmap over a range of ids, as it was left."""
    nbytes = lib.apt_unique_workspace_bytes(rng)
    if ws_name != "unique":
        # a bitmap of its own per id range: a captured graph that replays this call must find
        # the layout it was captured with, whatever ran on the shared bitmap in between
        ws_name = f"{ws_name}:{rng}"
    return STATE.workspace(ws_name, nbytes)


def _unique_workspace(rng, ws_name):
    """The same, zero."""
    ws = _unique_bitmap(rng, ws_name)
    if getattr(ws, "_apt_clean_range", None) != rng:
        # the bitmap has to be zero once per id range (the layout follows the range);
        # every call then leaves it zero again
        check(lib.apt_unique_workspace_init(_ptr(ws), ws.numel(), _stream()))
        ws._apt_clean_range = rng
    return ws


def _unique_enqueue(ids, n_dev, id_lo, id_hi, count_out, ws_name="unique"):
    """`ws_name` picks the cached bitmap: callers that alternate between id ranges give
    each range its own, so that none is cleared again on every call."""
    n = ids.numel()
    rng = int(id_hi) - int(id_lo)
    uniq = torch.empty(min(n, max(rng, 0)), dtype=torch.int64, device=ids.device)
    inv = torch.empty(n, dtype=torch.int64, device=ids.device)
    ws = _unique_workspace(rng, ws_name)
    check(lib.apt_unique_sorted(_ptr(ids), n, _ptr(n_dev), int(id_lo), int(id_hi), _ptr(ws), ws.numel(), _ptr(uniq),
                                _ptr(inv), _ptr(count_out), STATE.status_ptr(), _stream()))
    return uniq, inv


def _unique_ids(ids, n_dev, per, id_lo, id_hi, count_out, ws_name):
    """The distinct ids (n_dev: of n_dev * per); _unique_inverse has to follow with the same ids."""
    n = ids.numel()
    rng = int(id_hi) - int(id_lo)
    uniq = torch.empty(min(n, max(rng, 0)), dtype=torch.int64, device=ids.device)
    ws = _unique_workspace(rng, ws_name)
    ws._apt_clean_range = None      # until the inverse has it zero again
    check(lib.apt_unique_ids(_ptr(ids), n, _ptr(n_dev), int(per), int(id_lo), int(id_hi), _ptr(ws), ws.numel(), _ptr(uniq), _ptr(count_out),
                             STATE.status_ptr(), _stream()))
    return uniq


def _unique_inverse(ids, n_dev, per, id_lo, id_hi, ws_name, uniq=None, uniq_n=None, sizes=None, offsets=None, side=None, head=None,
                    head_n=None, all_out=None, look_up=False):
    """The inverse of _unique_ids, on side stream `side` (which the caller joins) or the current one. From the same launch:
    with `sizes` and `offsets` what _bucket leaves in a world of one rank, of the ids or of the distinct ones (`uniq`, whose count is uniq_n);
    with `head` the list concat_ids(head, head_n, uniq, uniq_n, all_out, look_up). Returns (inverse, permutation or None, list or None)."""
    rng = int(id_hi) - int(id_lo)
    ws = _unique_bitmap(rng, ws_name)
    try:
        if sizes is not None and STATE.shuffle_min_vids is None:
            raise RuntimeError("register_min_vids has not been called")
        n, dev = ids.numel(), ids.device
        inv = torch.empty(n, dtype=torch.int64, device=dev)
        n_uniq = 0 if uniq is None else uniq.numel()
        perm = None if sizes is None else torch.empty(n if uniq is None else n_uniq, dtype=torch.int64, device=dev)
        listed = None if head is None else torch.empty(head.numel() + n_uniq, dtype=torch.int64, device=dev)
        if perm is not None and perm.numel() == 0:
            sizes.zero_()
            offsets.zero_()
            sizes = offsets = None
        if listed is not None and listed.numel() == 0:
            all_out.zero_()
        with contextlib.nullcontext() if side is None else STATE.beside(side):
            check(lib.apt_unique_inverse(
                _ptr(ids), n, _ptr(n_dev), int(per), int(id_lo), int(id_hi), _ptr(ws), ws.numel(), _ptr(inv), _ptr(uniq), n_uniq, _ptr(uniq_n),
                _ptr(perm), _ptr(sizes), _ptr(offsets),
                _ptr(head), 0 if head is None else head.numel(), _ptr(head_n), _ptr(listed), _ptr(all_out),
                *(_row_tables() if look_up else (None, 0, 0, 0)), STATE.status_ptr(), _stream()))
    except BaseException:
        # the distinct ids' counts are still in the bitmap, which a captured graph may take next without looking
        if not torch.cuda.is_current_stream_capturing():
            lib.apt_unique_workspace_init(_ptr(ws), ws.numel(), _stream())
        raise
    ws._apt_clean_range = rng
    return inv, perm, listed


def concat_ids(a: torch.Tensor, na_dev: Optional[torch.Tensor], b: torch.Tensor, nb_dev: Optional[torch.Tensor],
               count_out: Optional[torch.Tensor], look_up: bool = False) -> torch.Tensor:
    """cat(a[:na], b[:nb]) with device-side lengths (None: the whole tensor); the result buffer holds
    a.numel() + b.numel() ids and the device word `count_out` receives na + nb. `look_up`: the ids are those of
    a gather, flag what it would flag."""
    out = torch.empty(a.numel() + b.numel(), dtype=torch.int64, device=a.device)
    check(lib.apt_concat_row_ids(_ptr(a), a.numel(), _ptr(na_dev), _ptr(b), b.numel(), _ptr(nb_dev), _ptr(out),
                                 _ptr(count_out), *(_row_tables() if look_up else (None, 0, 0, 0)), STATE.status_ptr(),
                                 _stream()))
    return out


def _owned_range():
    """Ids this rank can receive from a seed shuffle. On one machine these are
    the ids it owns; with several machines foreign ids are re-mapped to the
    sender itself (src/cuda/npc_kernel.cu:340-342), so any id may arrive."""
    s = STATE
    n_total = s.graph.num_total_nodes
    if s.node_size == s.world_size and s.shuffle_id_offset == 0 and s._min_vids_host is not None:
        lo = int(s._min_vids_host[s.rank])
        hi = int(s._min_vids_host[s.rank + 1])
        if s.rank == 0:
            lo = min(lo, 0)
        if s.rank == s.world_size - 1:
            hi = max(hi, n_total)
        return lo, hi
    return 0, n_total


def np_sample_and_shuffle(seeds: torch.Tensor, fanout: int) -> List[torch.Tensor]:
    """NPSampleAndShuffle, src/sampling.cc:52-69: [unique_frontier, neighbors,
    permutation, recv_offset, dev_offset, inverse_idx]."""
    recv, perm, recv_offset, dev_offset = shuffle_seeds(seeds)
    lo, hi = _owned_range()
    uniq, inverse_idx = unique_sorted(recv, lo, hi)
    neighbors = _sample(uniq, fanout)
    return [uniq, neighbors, perm, recv_offset, dev_offset, inverse_idx]


def sp_sample_shuffle_src(unique_src: torch.Tensor) -> List[torch.Tensor]:
    """SPSampleShuffleSrc, src/sampling.cc:151-157."""
    return list(shuffle_seeds(unique_src))


# ------------------------------------------------- SNP virtual nodes (SAGE / GCN)
SP_BASE = 10_000_000   # python/npc/sampler.py:181: virtual node = sender * SP_BASE + destination index


def _owner_args():
    s = STATE
    if s.shuffle_min_vids is None:
        raise RuntimeError("register_min_vids has not been called")
    node_beg = s.rank - s.rank % s.node_size
    return _ptr(s.shuffle_min_vids), s.world_size, int(s.shuffle_id_offset), s.rank, node_beg, node_beg + s.node_size


def src_to_vir(fanout: int, num_dst: int, src: torch.Tensor) -> torch.Tensor:
    """SrcToVir, src/sampling.cc:19-34: owner(src[i]) * num_dst + i // fanout."""
    src = _need_cuda(src, "src")
    out = torch.empty_like(src)
    check(lib.apt_src_to_vir(_ptr(src), src.numel(), int(fanout), int(num_dst), *_owner_args(), _ptr(out), _stream()))
    return out


def srcdst_to_vir(fanout: int, dst: torch.Tensor, src: torch.Tensor) -> torch.Tensor:
    """SrcDsttoVir, src/sampling.cc:36-50: destinations first, then the
    neighbours shifted by world_size * num_dst."""
    dst = _need_cuda(dst, "dst")
    src = _need_cuda(src, "src")
    out = torch.empty(dst.numel() + src.numel(), dtype=torch.int64, device=src.device)
    check(lib.apt_srcdst_to_vir(_ptr(dst), dst.numel(), _ptr(src), src.numel(), int(fanout), *_owner_args(),
                                _ptr(out), _stream()))
    return out


def vir_send_sizes(num_seeds: int, sorted_allnodes: torch.Tensor, unique_frontier: torch.Tensor,
                   shuffle_with_dst: int, with_offsets: bool = False):
    """Device tensor of the k = 2 (3 with destinations) sizes per receiver that
    SPSampleAndShuffle exchanges (src/sampling.cc:86-106)."""
    ws = STATE.world_size
    k = 3 if shuffle_with_dst else 2
    sizes = torch.empty(k * ws, dtype=torch.int64, device=sorted_allnodes.device)
    offs = torch.empty(k * ws + 1, dtype=torch.int64, device=sorted_allnodes.device) if with_offsets else None
    check(lib.apt_vir_send_sizes(_ptr(sorted_allnodes), sorted_allnodes.numel(), None, _ptr(unique_frontier),
                                 unique_frontier.numel(), None, ws, int(num_seeds), None, int(bool(shuffle_with_dst)),
                                 _ptr(offs), _ptr(sizes), _stream()))
    return (sizes, offs) if with_offsets else sizes


def sp_pack_frontier(sorted_vir: torch.Tensor, sorted_ids: torch.Tensor, num_dst: int) -> torch.Tensor:
    """rank * SP_BASE * N + (sorted_vir % num_dst) * N + sorted_ids, the packed
    (sender, destination index, neighbour id) of python/npc/sampler.py:296-300."""
    out = torch.empty_like(sorted_ids)
    check(lib.apt_sp_pack_frontier(_ptr(sorted_vir), _ptr(sorted_ids), sorted_ids.numel(), int(num_dst), STATE.rank,
                                   SP_BASE, int(STATE.graph.num_total_nodes), _ptr(out), _stream()))
    return out


def _cumsum_cpu(sizes: torch.Tensor) -> torch.Tensor:
    return sizes.cumsum(0) if sizes.numel() else sizes


def sp_sample_and_shuffle(num_dst: int, send_frontier: torch.Tensor, sorted_allnodes: torch.Tensor,
                          unique_frontier: torch.Tensor, shuffle_with_dst: int) -> List[torch.Tensor]:
    """SPSampleAndShuffle, src/sampling.cc:71-149: [vir_src, ori_src, send_sizes,
    recv_sizes] or, with destinations, [recv_dst, vir_src, ori_src, send_sizes,
    recv_sizes]; the size vectors are CPU int64 as in the reference."""
    send_frontier = _need_cuda(send_frontier, "send_frontier")
    sorted_allnodes = _need_cuda(sorted_allnodes, "sorted_allnodes")
    unique_frontier = _need_cuda(unique_frontier, "unique_frontier")
    s = STATE
    ws = s.world_size
    with_dst = int(bool(shuffle_with_dst))
    k = 3 if with_dst else 2
    ex = _exchange()
    send_sizes_dev = vir_send_sizes(num_dst, sorted_allnodes, unique_frontier, with_dst)
    recv_sizes_dev = torch.empty_like(send_sizes_dev)
    steps = torch.arange(1, ws + 1, dtype=torch.int64) * k
    ex.alltoall(send_sizes_dev, recv_sizes_dev, steps, steps, 1)
    both = torch.stack([send_sizes_dev, recv_sizes_dev]).cpu()
    send_sizes, recv_sizes = both[0].contiguous(), both[1].contiguous()
    n_total = int(s.graph.num_total_nodes)
    dev = send_frontier.device
    if with_dst:
        sd, rd = send_sizes[0::3], recv_sizes[0::3]
        ss, rs = send_sizes[1::3], recv_sizes[1::3]
        n_sd, n_rd, n_rs = int(sd.sum()), int(rd.sum()), int(rs.sum())
        recv_all = torch.empty(n_rd + n_rs, dtype=torch.int64, device=dev)
        ex.alltoall(send_frontier[:n_sd], recv_all[:n_rd], _cumsum_cpu(sd), _cumsum_cpu(rd), 1)
        ex.alltoall(send_frontier[n_sd:], recv_all[n_rd:], _cumsum_cpu(ss), _cumsum_cpu(rs), 1)
        recv_src = recv_all[n_rd:]
    else:
        ss, rs = send_sizes[0::2], recv_sizes[0::2]
        n_rs = int(rs.sum())
        recv_src = torch.empty(n_rs, dtype=torch.int64, device=dev)
        ex.alltoall(send_frontier, recv_src, _cumsum_cpu(ss), _cumsum_cpu(rs), 1)
    vir_src = torch.empty(n_rs, dtype=torch.int64, device=dev)
    ori_src = torch.empty(n_rs, dtype=torch.int64, device=dev)
    check(lib.apt_sp_unpack_frontier(_ptr(recv_src), n_rs, None, n_total, _ptr(vir_src), _ptr(ori_src), _stream()))
    if with_dst:
        return [recv_all[:n_rd], vir_src, ori_src, send_sizes, recv_sizes]
    return [vir_src, ori_src, send_sizes, recv_sizes]


def sp_feat_shuffle(inputs: torch.Tensor, send_sizes: torch.Tensor, recv_sizes: torch.Tensor, total_recv_size: int,
                    expand: int, shuffle_with_dst: int) -> torch.Tensor:
    """SPFeatShuffle, src/feat_shuffle.cc:32-52: rows of `expand` elements; per
    peer q the last of its k sizes (partial sums per virtual node), preceded,
    with destinations, by sizes[3 q] destination rows for every q."""
    ex = _exchange()
    if ex.name == "local":
        return _native.sp_feat_shuffle_local(inputs, send_sizes, recv_sizes, int(total_recv_size), int(expand), bool(shuffle_with_dst))
    if inputs.dtype not in _DTYPE_CODE:
        raise RuntimeError(f"sp_feat_shuffle: unsupported dtype {inputs.dtype}")
    inputs = _need_cuda(inputs, "inputs", dtype=None)
    expand = int(expand)
    rows = inputs.numel() // expand
    flat = inputs.view(rows, expand)
    out = torch.empty((int(total_recv_size), expand), dtype=inputs.dtype, device=inputs.device)
    send_sizes, recv_sizes = send_sizes.cpu(), recv_sizes.cpu()
    if shuffle_with_dst:
        sd, rd = send_sizes[0::3], recv_sizes[0::3]
        sv, rv = send_sizes[2::3], recv_sizes[2::3]
        n_sd, n_rd = int(sd.sum()), int(rd.sum())
        if n_sd + int(sv.sum()) != rows or n_rd + int(rv.sum()) != int(total_recv_size):
            raise RuntimeError("sp_feat_shuffle: sizes do not add up to the rows given")
        ex.alltoall(flat[:n_sd], out[:n_rd], _cumsum_cpu(sd), _cumsum_cpu(rd), expand)
        ex.alltoall(flat[n_sd:], out[n_rd:], _cumsum_cpu(sv), _cumsum_cpu(rv), expand)
    else:
        sv, rv = send_sizes[1::2], recv_sizes[1::2]
        if int(sv.sum()) != rows or int(rv.sum()) != int(total_recv_size):
            raise RuntimeError("sp_feat_shuffle: sizes do not add up to the rows given")
        ex.alltoall(flat, out, _cumsum_cpu(sv), _cumsum_cpu(rv), expand)
    return out


# ------------------------------------------- NFP (feature dimension partitioned)
def mp_sample_shuffle(seeds: torch.Tensor, unique_frontier: torch.Tensor, coo_row: torch.Tensor) -> List[torch.Tensor]:
    """MPSampleShuffle, src/sampling.cc:195-239: every rank receives every
    rank's frontier and relabelled rows. [recv_frontier, recv_coo_row,
    [seeds_size] (cpu), recv_seeds_size (cpu), recv_frontier_size (cpu),
    recv_coo_size (cpu)]."""
    unique_frontier = _need_cuda(unique_frontier, "unique_frontier")
    coo_row = _need_cuda(coo_row, "coo_row")
    ws = STATE.world_size
    ex = _exchange()
    mine = torch.tensor([[seeds.numel(), unique_frontier.numel(), coo_row.numel()]], dtype=torch.int64,
                        device=unique_frontier.device)
    sizes = ex.allbroadcast(mine, [1] * ws).cpu()                       # [ws, 3]
    recv_seeds_size = sizes[:, 0].contiguous()
    recv_frontier_size = sizes[:, 1].contiguous()
    recv_coo_size = sizes[:, 2].contiguous()
    recv_frontier = ex.allbroadcast(unique_frontier.view(-1, 1), recv_frontier_size.tolist()).view(-1)
    recv_coo_row = ex.allbroadcast(coo_row.view(-1, 1), recv_coo_size.tolist()).view(-1)
    return [recv_frontier, recv_coo_row, torch.tensor([seeds.numel()]), recv_seeds_size, recv_frontier_size,
            recv_coo_size]


def mp_feat_shuffle_fwd(inputs: torch.Tensor, send_size: torch.Tensor, recv_size: torch.Tensor,
                        feat_dim: int) -> torch.Tensor:
    """MPFeatShuffleFwd, src/feat_shuffle.cc:54-64 (a reduce-scatter): rows
    [off[r], off[r] + send_size[r]) of every rank's inputs are summed on rank r,
    which gets recv_size rows. The sum runs over the ranks in rank order in fp32."""
    if inputs.dtype not in _DTYPE_CODE:
        raise RuntimeError(f"mp_feat_shuffle_fwd: unsupported dtype {inputs.dtype}")
    inputs = _need_cuda(inputs, "inputs", dtype=None)
    feat_dim = int(feat_dim)
    flat = inputs.view(inputs.numel() // feat_dim, feat_dim)
    send_size = send_size.cpu().to(torch.int64).view(-1)
    mine = int(recv_size.view(-1)[0])
    if int(send_size.sum()) != flat.shape[0] or int(send_size[STATE.rank]) != mine:
        raise RuntimeError("mp_feat_shuffle_fwd: sizes do not match the rows given")
    return _exchange().reduce_scatter(flat, send_size, mine)


def mp_feat_shuffle_bwd(inputs: torch.Tensor, send_size: torch.Tensor, recv_size: torch.Tensor,
                        feat_dim: int) -> torch.Tensor:
    """MPFeatShuffleBwd, src/feat_shuffle.cc:66-79 (an all-gather of blocks of
    different lengths): every rank receives every rank's rows in rank order."""
    inputs = _need_cuda(inputs, "inputs", dtype=None)
    feat_dim = int(feat_dim)
    flat = inputs.view(inputs.numel() // feat_dim, feat_dim)
    if int(send_size.view(-1)[0]) != flat.shape[0]:
        raise RuntimeError("mp_feat_shuffle_bwd: send_size does not match the rows given")
    return _exchange().allbroadcast(flat, [int(x) for x in recv_size.view(-1).tolist()])


# ---------------------------------------------------------------------- gather
def load_subtensor(node_id: torch.Tensor) -> torch.Tensor:
    """LoadSubtensor, src/load_subtensor.cc:19-40: rows of the GPU cache or,
    on a miss, of the page-locked host table, in one call."""
    f = STATE.feat
    if f.feat_pos_map is None:
        raise RuntimeError("cache_feats_shared has not been called")
    ahead = STATE.prefetched
    if ahead is not None:
        STATE.prefetched = None
        if ahead.serves(node_id):
            if ahead.pending is not None:
                ahead.pending.order_current_stream()
            return ahead.rows
    return _native.gather(node_id, f.feat_pos_map, f.dev_feats, f.uva_feats, f.num_total_nodes, f.feat_dim_offset,
                          STATE.words())


def _gather_enqueue(node_id: torch.Tensor, n_dev: Optional[torch.Tensor], out: Optional[torch.Tensor] = None,
                    first_dev: Optional[torch.Tensor] = None, ws_name: str = "gather", beside: bool = False,
                    publish=None) -> torch.Tensor:
    """Enqueues the gather of rows [first_dev, n_dev) of node_id (device words; None: 0 and
    node_id.numel()) into `out` (allocated here when None). Calls that may overlap on the GPU
    need workspaces of their own (`ws_name`). `beside`: on a few blocks, beside other kernels. `publish`: the
    arguments of apt_publish_tagged but for the stream; the words leave beside the rows."""
    f = STATE.feat
    n = node_id.numel()
    esz = f.dev_feats.element_size()
    if out is None:
        out = torch.empty((n, f.rank_feat_dim), dtype=f.dev_feats.dtype, device=node_id.device)
    if publish is not None:
        check(lib.apt_gather_rows_publish(
            _ptr(node_id), n, _ptr(n_dev), _ptr(first_dev), _ptr(f.feat_pos_map), f.num_total_nodes,
            _ptr(f.dev_feats), f.dev_feats.shape[0], f.rank_feat_dim * esz,
            _ptr(f.uva_feats), f.uva_feats.shape[0], f.feat_dim * esz, f.feat_dim_offset * esz,
            _ptr(out), STATE.status_ptr(), *publish, _stream()))
        return out
    nbytes = lib.apt_gather_workspace_bytes(n)
    ws = STATE.workspace(ws_name, nbytes)
    launch, counts = (lib.apt_gather_rows_beside, (_ptr(n_dev),)) if beside else \
        (lib.apt_gather_rows_from, (_ptr(n_dev), _ptr(first_dev)))
    check(launch(
        _ptr(node_id), n, *counts, _ptr(f.feat_pos_map), f.num_total_nodes,
        _ptr(f.dev_feats), f.dev_feats.shape[0], f.rank_feat_dim * esz,
        _ptr(f.uva_feats), f.uva_feats.shape[0], f.feat_dim * esz, f.feat_dim_offset * esz,
        _ptr(out), _ptr(ws), ws.numel(), STATE.status_ptr(), _stream()))
    return out


def cpu_load_subtensor(node_id: torch.Tensor) -> torch.Tensor:
    """CPULoadSubtensor, src/load_subtensor.cc:10-17: host table only, on the
    CPU, as the reference does it (two index_selects)."""
    f = STATE.feat
    pos = -f.cpu_feat_pos_map.index_select(0, node_id.cpu()) - 2
    table = f.uva_feats if not f.uva_feats.is_cuda else f.uva_feats.cpu()
    return table.index_select(0, pos)


# -------------------------------------------------------------- feature shuffle
def feat_shuffle(inputs: torch.Tensor, send_offset: torch.Tensor, recv_offset: torch.Tensor,
                 permutation: torch.Tensor, feat_dim: int, fwd_flag: int) -> torch.Tensor:
    """FeatShuffle, src/feat_shuffle.cc:9-30. Offsets are CPU int64 inclusive
    cumulative row counts. fwd: rows travel to the ranks that asked for them
    and come out in the asker's original seed order (``buf[permutation]``);
    bwd: rows are scattered by permutation and travel back."""
    ex = _exchange()
    if ex.name == "local":
        return _native.feat_shuffle_local(inputs, recv_offset, permutation, int(feat_dim), bool(fwd_flag))
    if inputs.dtype not in _DTYPE_CODE:
        raise RuntimeError(f"feat_shuffle: unsupported dtype {inputs.dtype}")
    inputs = _need_cuda(inputs, "inputs", dtype=None)
    permutation = _need_cuda(permutation, "permutation")
    rows_in = inputs.numel() // int(feat_dim)
    return ex.exchange_rows(inputs.view(rows_in, int(feat_dim)), send_offset, recv_offset, permutation, bool(fwd_flag))


def alltoall(input: torch.Tensor, output: torch.Tensor, send_offset: torch.Tensor, recv_offset: torch.Tensor,
             expand: int = 1, comm_type: int = 0) -> None:
    """AlltoAll, src/ops/collective.cc:252-266: in place into `output`; any
    dtype (the reference silently ignores everything but int64/fp32)."""
    _exchange().alltoall(_need_cuda(input, "input", dtype=None), output, send_offset, recv_offset, int(expand))


# ---------------------------------------------------------------- SpMM / SDDMM
def _spmm(op, coo_row, coo_col, inp, edata, coo_offset, input_offset, output_offset):
    return _native.spmm(op, coo_row, coo_col, inp, edata, coo_offset, input_offset, output_offset)


def spmm_copy_u_sum(coo_row, coo_col, input, coo_offset, input_offset, output_offset):
    """CopyUSum, src/spmm.cc:9-19."""
    return _spmm(0, coo_row, coo_col, input, None, coo_offset, input_offset, output_offset)


def spmm_copy_e_sum(coo_row, coo_col, input, coo_offset, output_offset):
    """CopyESum, src/spmm.cc:21-29: `input` holds one row per edge."""
    return _spmm(1, coo_row, coo_col, None, input, coo_offset, None, output_offset)


def spmm_u_mul_e_sum(coo_row, coo_col, input, edata, coo_offset, input_offset, output_offset, ref_quirk_add=False):
    """UMulESum, src/spmm.cc:31-42: sum over edges of input[src] * edata[e].
    The reference's kernel adds instead of multiplying (src/cuda/spmm.cu:78);
    ref_quirk_add=True reproduces that."""
    return _spmm(3 if ref_quirk_add else 2, coo_row, coo_col, input, edata, coo_offset, input_offset, output_offset)


def sddmm_u_add_v(coo_row, coo_col, lhs, rhs, coo_offset, lhs_offset, rhs_offset):
    """UAddV, src/sddmm.cc:9-19."""
    return _native.sddmm(0, coo_row, coo_col, lhs, rhs, coo_offset, lhs_offset, rhs_offset)


def sddmm_u_mul_v(coo_row, coo_col, lhs, rhs, coo_offset, lhs_offset, rhs_offset):
    """UMulV, src/sddmm.cc:21-31."""
    return _native.sddmm(1, coo_row, coo_col, lhs, rhs, coo_offset, lhs_offset, rhs_offset)


def gat_edge_softmax_sum(coo_row, coo_col, ft, el, er, num_dst: int, negative_slope: float = 0.2,
                         return_attention: bool = False):
    """One sampled block of a GAT layer: u_add_v(el, er) -> leaky_relu -> edge_softmax -> u_mul_e(ft, a) summed per destination (the DGL calls of
    python/npc/model/gatconv.py:113-124). ft [num_src, H, Dh] or [num_src, H*Dh],
    el [num_src, H(,1)], er [num_dst, H(,1)]; edges grouped by destination.
    Returns out [num_dst, H, Dh] (and the attention [E, H, 1])."""
    out, attn = _native.gat_forward(coo_row, coo_col, ft, el, er, int(num_dst), float(negative_slope),
                                    bool(return_attention), STATE.words())
    return (out, attn) if return_attention else out


def gat_edge_softmax_sum_backward(coo_row, coo_col, ft, el, er, grad_out, negative_slope: float = 0.2):
    """Gradients of gat_edge_softmax_sum with respect to ft, el and er for
    grad_out [num_dst, H, Dh]: the edge part over the destinations (softmax and
    leaky_relu backward per edge, grad_er, and grad_el added up in fp32 by
    reductions), then one walk over the edges grouped by source for grad_ft. Both
    source-side sums run in an order that the GPU's scheduling decides, so they
    repeat themselves within rounding and not bit for bit. Returns (grad_ft,
    grad_el, grad_er) shaped like ft, el, er."""
    return _native.gat_backward(coo_row, coo_col, ft, el, er, grad_out, float(negative_slope), STATE.words())


class GATEdgeSoftmaxSum:
    """gat_edge_softmax_sum with its backward, for use inside a model:
    ``out = GATEdgeSoftmaxSum.apply(coo_row, coo_col, ft, el, er, num_dst, slope)``
    (an autograd function on the C++ side)."""

    @staticmethod
    def apply(coo_row, coo_col, ft, el, er, num_dst, negative_slope=0.2):
        return _native.gat_apply(coo_row, coo_col, ft, el, er, int(num_dst), float(negative_slope), STATE.words())


# ------------------------------------------------------------------ row movers
def rows_gather(inp: torch.Tensor, index: torch.Tensor) -> torch.Tensor:
    """out[i] = inp[index[i]] for 2-D inp (the model's h[inverse_idx],
    python/npc/model/sage_model.py:67)."""
    return _native.rows_gather(inp, index)


def rows_scatter(inp: torch.Tensor, index: torch.Tensor, num_out_rows: int) -> torch.Tensor:
    """out[index[i]] = inp[i]; rows of out not named by index are zero."""
    return _native.rows_scatter(inp, index, int(num_out_rows))
