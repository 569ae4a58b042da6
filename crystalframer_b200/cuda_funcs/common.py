"""Helpers shared by the autograd Functions."""
import time
import weakref

import torch

from .. import _lib

_csr_cache = {}


def csr_offsets(edge_ij_e, N):
    """e_start (N+1): first pair of every query atom.  The reference rebuilds it with
    scatter_add + cumsum in each Function (models/cuda_funcs/fused_dpa.py:24-26); here it is
    computed once per pair list and cached while that tensor is alive and unmodified."""
    key = id(edge_ij_e)
    hit = _csr_cache.get(key)
    if hit is not None:
        ref, version, n, out = hit
        if ref() is edge_ij_e and version == edge_ij_e._version and n == N:
            return out
    E = edge_ij_e.shape[1]
    out = torch.empty(N + 1, dtype=torch.int64, device=edge_ij_e.device)
    _lib.invoke("cfb200_csr_offsets", 1, edge_ij_e.device, _lib.iptr(edge_ij_e), E, N, _lib.iptr(out))
    if len(_csr_cache) > 64:
        for k in [k for k, v in _csr_cache.items() if v[0]() is None]:
            del _csr_cache[k]
    _csr_cache[key] = (weakref.ref(edge_ij_e), edge_ij_e._version, N, out)
    return out


def register_csr(edge_ij_e, N, e_start):
    """Lets a caller that already holds the offsets (cfb200_edge_index) seed the cache."""
    _csr_cache[id(edge_ij_e)] = (weakref.ref(edge_ij_e), edge_ij_e._version, N, e_start)


def f32c(t):
    """Contiguous float32 data of a tensor on the 16-byte grid: the kernels read 128 bits at a time, and a contiguous
    slice of a tensor may begin anywhere."""
    if t is None:
        return None
    t = t.detach().contiguous().float()
    return t.clone() if t.data_ptr() & 15 else t


def kept(*tensors):
    """What a result that is kept for these tensors holds to tell whether it still stands (unchanged): the tensors, or aliases of
    them, so that no other tensor can take their place in memory, and where that is and the version of its contents (none for
    tensors that do not count theirs: they are never found unchanged)."""
    return tuple((t, t.data_ptr(), None if t.is_inference() else t._version) for t in tensors)


def unchanged(entries, *tensors):
    for (t, address, version), u in zip(entries, tensors):
        if version is None or u.is_inference() or u.data_ptr() != address or u._version != version:
            return False
        if u is not t and (u.shape != t.shape or u.stride() != t.stride() or u.dtype != t.dtype):
            return False
    return True


_pair_cache = {}
PAIR_LIST_BYTES_PER_PAIR = 5 * 128 * 4   # five planes of 128 floats: 2.5 KB of translation list per pair
PAIR_LIST_MAX_PAIRS = 4_000_000          # hard cap (10 GB); below it the list also has to fit a quarter of the free memory


_FREE_MEMORY = {}          # device -> (free bytes at the last query, when that was)
FREE_MEMORY_SECONDS = 10.0


def pair_list_fits(num_pairs, device):
    """Whether the per-pair translation lists of a batch may be built: the batch's lists (2.5 KB per pair, e.g. 133 MB
    for 52 k pairs, 3.6 GB for the 1.4 M pairs of a large-cell batch) must stay under a quarter of the device memory
    that is free right now and under the hard cap; otherwise the kernels sweep the translations instead."""
    if num_pairs > PAIR_LIST_MAX_PAIRS:
        return False
    need = num_pairs * PAIR_LIST_BYTES_PER_PAIR
    # The driver query can take tens of milliseconds (41 ms measured; asked every 64 batches it was a third of a training
    # step of 8 crystals): an answer of the last ten seconds serves requests far below it.
    key = (device.type, device.index)
    now = time.monotonic()
    free, asked = _FREE_MEMORY.get(key, (0, 0.0))
    if need > free // 32 or now - asked > FREE_MEMORY_SECONDS:
        free = torch.cuda.mem_get_info(device)[0]
        _FREE_MEMORY[key] = (free, now)
    return need <= free // 4


def allocate_pair_list(num_pairs, device):
    """Room for a batch's translation lists, or None where they do not fit (also where the memory went since it was asked
    for)."""
    if not pair_list_fits(num_pairs, device):
        return None
    try:
        return torch.empty((num_pairs, 5, 128), dtype=torch.float32, device=device)
    except torch.OutOfMemoryError:
        _FREE_MEMORY.pop((device.type, device.index), None)
        return None


def pair_geometry(rpos_ij_e, tvecs_n, batch_i, edge_ij_e, cutoff):
    """(pair_cache, pair_list, cache_range): which lattice translations of every pair are near, and how
    near -- the nearest non-zero image, the smallest squared distance, all translations sorted by distance.
    Pure geometry, identical for every head and layer, so it is computed on the first call that sees a
    batch's relative positions and kept while that tensor is alive and it, the cells, the atoms' crystals and
    the pair list are what they were; the reference redoes this search inside every kernel launch.  Returns (None, None, 0) when no range can be fixed up front."""
    from .kernel_manager import KernelManager
    cfg = KernelManager.config
    if cfg is None or rpos_ij_e is None or edge_ij_e.shape[1] == 0:
        return None, None, 0
    rng = int(cfg.lattice_range if cutoff == 0.0 else cfg.minimum_range)
    if rng <= 0:
        return None, None, 0
    key = id(rpos_ij_e)
    hit = _pair_cache.get(key)
    if hit is not None and hit[0]() is rpos_ij_e and hit[1] == rng and unchanged(hit[4], rpos_ij_e, tvecs_n, batch_i, edge_ij_e):
        return hit[2], hit[3], rng
    _pair_cache.pop(key, None)
    dev = rpos_ij_e.device
    pos, tv = f32c(rpos_ij_e), f32c(tvecs_n)
    batch, edges = batch_i.contiguous(), edge_ij_e.contiguous()
    N, E = batch.shape[0], edges.shape[1]
    cache = torch.empty((E, 4), device=dev, dtype=torch.float32)
    plist = None
    if (2 * rng + 1) ** 3 <= 128:
        plist = allocate_pair_list(E, dev)
    _lib.invoke("cfb200_pair_cache", 2, dev, _lib.ptr(pos), _lib.ptr(tv), _lib.iptr(batch), _lib.iptr(edges), N, E, rng,
                _lib.ptr(cache), _lib.ptr(plist))
    for k in [k for k, v in _pair_cache.items() if v[0]() is None]:      # lists are large: drop dead batches at once
        del _pair_cache[k]
    # (aliases: the entry goes when the positions do, and a caller's pair list may hold on to those)
    _pair_cache[key] = (weakref.ref(rpos_ij_e), rng, cache, plist,
                        kept(*(t.detach() for t in (rpos_ij_e, tvecs_n, batch_i, edge_ij_e))))
    return cache, plist, rng
