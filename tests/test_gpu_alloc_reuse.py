"""cq_malloc / cq_free: freed blocks are handed out again, bounded in size, and never twice."""
import numpy as np
import pytest

from candy_b200 import abi
from candy_b200.backend import CudaDevice

pytestmark = pytest.mark.gpu


@pytest.fixture()
def fresh():
    d = CudaDevice(0)
    yield d
    d.close()


@pytest.mark.parametrize("nbytes,kept", [(1, True), (512, True), (513, True), (16 << 20, True), ((16 << 20) + 1, False)])
def test_freed_block_is_reused_up_to_the_limit(fresh, nbytes, kept):
    p = fresh.malloc(nbytes)
    fresh.free(p)
    if kept:
        assert fresh._lib.cq_free(fresh.ctx, p) != abi.OK  # freed before: not the caller's any more
    q, r = fresh.malloc(nbytes), fresh.malloc(nbytes)
    assert q.value != r.value
    if kept:
        assert q.value == p.value
    fresh.free(q)
    fresh.free(r)


def test_kept_blocks_are_bounded_and_sizes_fit(fresh):
    ps = [fresh.malloc(12 << 20) for _ in range(7)]
    for p in ps:
        fresh.free(p)
    again = [fresh.malloc(12 << 20).value for _ in range(7)]
    assert len(set(again)) == 7
    small = fresh.malloc(4096)  # a block more than twice the size is not taken
    fresh.free(small)
    a, b = fresh.malloc(1024), fresh.malloc(2500)
    assert a.value != small.value and b.value == small.value


def test_contents_survive_reuse_in_flight(fresh):
    """A block freed right after a launch that reads it: the next owner's writes come after that launch."""
    n = 1 << 20
    src = np.arange(n, dtype=np.float32)
    out = fresh.alloc(n)
    for i in range(20):
        a = fresh.storage_from_slice(src + i)
        abi.check(fresh.ctx, fresh._lib.cq_memcpy_d2d(fresh.ctx, out.ptr, a.ptr, 4 * n), "copy")
        del a
        b = fresh.zeros(n)
        assert (out.data() == src + i).all()
        del b
