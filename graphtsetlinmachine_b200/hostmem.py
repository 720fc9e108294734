"""Result arrays in recycled page-locked memory.

A result of a few megabytes in a fresh numpy array costs a page fault per page and a copy out of a staging buffer; in
page-locked memory the copy engine writes it directly, in the time of the transfer.  Page-locking is slow (0.5 ms per MB),
so the memory of an array that nobody refers to any more is kept for the next result, and a block is locked only for
every eighth array of a size that is asked for: a program's first results are ordinary arrays, and what locking costs is
spread over many.  Free blocks are given back when the last model is closed, blocks in use when their arrays go after that.

An array in a block does not own its data, which shows in ``flags.owndata`` and in that it cannot be resized in place; a copy
of it can.
"""

import collections
import ctypes as C
import threading
import weakref

import numpy as np

from . import _lib

SMALLEST, LARGEST = 64 << 10, 16 << 20      # bytes of an array that is worth it / that is not too much to lock
MOST = 128 << 20                            # bytes locked at a time, arrays in use included

PER_BLOCK = 8                               # arrays of a size class asked for, for every block that may be locked

_asked = collections.Counter()                          # size class -> arrays asked for
_blocks = collections.Counter()                         # size class -> blocks locked
_free = collections.defaultdict(collections.deque)      # size class -> addresses
_lock = threading.Lock()
_locked = 0
_models = set()                                         # handles of open models (set operations are atomic)
_keep = True                                            # blocks that come back are kept: not once the last model has closed


def _size_class(nbytes):
    """Next size of the form 2^k or 1.5 * 2^k: at most a third is unused."""
    size = 1 << (nbytes - 1).bit_length()
    return size * 3 // 4 if nbytes <= size * 3 // 4 else size


def _give_back(address, size):
    _free[size].append(address)             # atomic: may run in the garbage collector of any thread
    if not _keep:
        _drain()


def _drain():
    """Frees unused blocks.  Not while another thread, or the code that the garbage collector interrupted, is at it: they then
    wait for the next occasion."""
    if _lock.acquire(blocking=False):
        try:
            _drain_locked(0)
        finally:
            _lock.release()


def _drain_locked(limit):
    """Frees unused blocks until at most `limit` bytes are locked; the caller holds the lock."""
    global _locked
    for size, blocks in list(_free.items()):
        while blocks and _locked > limit:
            try:
                address = blocks.popleft()
            except IndexError:
                break
            _lib.load().gtm_host_free(address)
            _locked -= size
            _blocks[size] -= 1


def model_opened(handle):
    _models.add(handle)


def model_closed(handle):
    """May run in the garbage collector of any thread."""
    global _keep
    _models.discard(handle)
    if not _models:
        _keep = False
        _drain()


def _take(size):
    """Address of a free block, or a newly locked one while the limit allows; 0 when it does not."""
    global _locked, _keep
    try:
        return _free[size].popleft()
    except IndexError:
        pass
    lib = _lib.load()
    with _lock:
        if (_blocks[size] + 1) * PER_BLOCK > _asked[size]:
            return 0
        _drain_locked(MOST - size)          # free blocks of other sizes make room
        if _locked + size > MOST:
            return 0
        out = C.c_void_p()
        if lib.gtm_host_alloc(size, C.byref(out)) != 0:
            return 0
        _locked += size
        _blocks[size] += 1
        _keep = True
        return out.value


def empty(shape, dtype):
    """Like ``numpy.empty``."""
    nbytes = int(np.prod(shape, dtype=np.int64)) * np.dtype(dtype).itemsize
    if not SMALLEST <= nbytes <= LARGEST:
        return np.empty(shape, dtype=dtype)
    size = _size_class(nbytes)
    _asked[size] += 1
    address = _take(size)
    if not address:
        return np.empty(shape, dtype=dtype)
    block = (C.c_ubyte * size).from_address(address)    # every array made from it keeps it alive
    weakref.finalize(block, _give_back, address, size).atexit = False
    return np.frombuffer(block, dtype=dtype, count=nbytes // np.dtype(dtype).itemsize).reshape(shape)
