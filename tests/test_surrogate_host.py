"""The surrogates' host side without a GPU, on a stand-in for the CUDA runtime."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import fake_cuda


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return fake_cuda.build(tmp_path_factory.mktemp("fake_cuda"))


@pytest.fixture(autouse=True)
def _reset(lib):
    lib.fake_reset()
    yield
    lib.fake_reset()


@pytest.mark.parametrize("in_dim,rows,device", [(1, 100_000, 0), (48, 5000, 0), (49, 334, 0), (49, 335, 1), (97, 168, 0),
                                                (97, 169, 1), (256, 1000, 1)])
def test_narrow_or_small_training_sets_take_the_host_statistics(lib, in_dim, rows, device):
    """The device's chain of additions takes as long for one column as for a hundred."""
    m = fake_cuda.Model(lib, "ta3s" if in_dim == 97 else "ta3w", in_dim)
    lib.fake_reset()
    assert m.set_data(rows) == 0
    assert m.launches("column_stats_kernel") == device
    m.close()


KINDS = [("ta3s", 97), ("ta3w", 97)]


@pytest.mark.parametrize("kind,in_dim", KINDS)
@pytest.mark.parametrize("nth", [0, 1, 2])
def test_no_memory_for_more_rows_leaves_room_for_none(lib, kind, in_dim, nth):
    """The buffers of the rows grow one by one, each freed before its larger one is allocated: when one of them
    fails, fewer rows need fresh buffers too, and no kernel gets a null pointer."""
    m = fake_cuda.Model(lib, kind, in_dim)
    assert m.set_data(100) == 0
    lib.fake_fail(b"cudaMalloc", nth)
    assert m.set_data(3000) == 1
    lib.fake_reset()
    x, out = {"ta3s": (0, 4), "ta3w": (0, 5)}[kind]                 # pack_kernel's rows and result
    for arg in (x, out):
        lib.fake_capture(b"pack_kernel", arg, 8)
        assert m.predict(60) == 0
        assert m.captured(np.uint64)[0] != 0
        lib.fake_reset()
    m.close()


@pytest.mark.parametrize("kind,in_dim", KINDS)
@pytest.mark.parametrize("call,rows", [("predict", 40), ("predict", 3000), ("set_data", 40), ("set_data", 3000),
                                       ("set_data_standardized", 3000)])
def test_a_failed_call_leaves_no_training_set_behind(lib, kind, in_dim, call, rows):
    """Prediction rows and a new training set take the old one's place on the device. Whichever runtime call
    fails on the way, training afterwards is refused, unless nothing had been touched yet."""
    def run(m):
        return m.predict(rows) if call == "predict" else m.set_data(rows, call)

    m = fake_cuda.Model(lib, kind, in_dim)
    assert m.set_data(100) == 0 and m.train(1, 50) == 0
    lib.fake_reset()
    assert run(m) == 0
    steps = m.log()
    m.close()
    seen: dict[str, int] = {}
    for step in steps:
        nth = seen[step] = seen.get(step, 0) + 1
        if step in ("cudaFree", "cudaFreeHost"):            # (their results are not looked at)
            continue
        m = fake_cuda.Model(lib, kind, in_dim)
        assert m.set_data(100) == 0 and m.train(1, 50) == 0
        lib.fake_reset()
        lib.fake_fail(step.encode(), nth - 1)
        assert run(m) == 1, (step, nth)
        untouched = step in ("cudaSetDevice", "cudaHostAlloc")
        lib.fake_reset()
        for again in (m.train(1, 50), m.gradients()):
            assert again == (0 if untouched else 1), (step, nth)
            assert untouched or "no data" in m.error()
        assert m.set_data(60) == 0 and m.train(1, 50) == 0   # and a new set is taken
        m.close()


def test_a_status_that_no_call_has_read_is_not_the_next_calls(lib):
    """A bit that a kernel set stays when the call fails before it reads the status (here at the launch behind
    it); the next call starts from zero."""
    m = fake_cuda.Model(lib, "ta3s")
    assert m.set_data(100) == 0 and m.gradients() == 0
    status = C.cast(lib.fake_block(4), C.POINTER(C.c_uint32))       # the only block of one word
    lib.fake_reset()
    for fails, nth, call in (("cudaLaunchKernel", 1, m.gradients), ("cudaMemcpyAsync", 0, m.gradients),
                             ("cudaStreamSynchronize", 0, m.gradients), ("cudaMemcpyAsync", 2, lambda: m.train(1, 50))):
        lib.fake_fail(fails.encode(), nth)
        assert call() == 1
        status[0] = 1                                                # as the kernel before it would have
        lib.fake_reset()
        assert m.gradients() == 0, (fails, m.error())
        assert status[0] == 0
    status[0] = 1                                                    # found by the call itself: reported once
    assert m.gradients() == 1 and "timed out" in m.error()
    assert m.gradients() == 0
    m.close()


def _corrections(m, epochs, batch, rows):
    """The first and last step's bias correction 1 - 0.999^t of a training call that succeeds."""
    lib = m.lib
    if m.kind == "ta3w":                                             # last_kernel's Adam: three pointers, six floats, c2
        lib.fake_capture(b"last_kernel", 2, 48)
        assert m.train(epochs, batch) == 0
        n = m.launches("last_kernel")
        return m.captured(np.float32, 0)[11], m.captured(np.float32, n - 1)[11]
    if batch > 1024:                                                 # adam_kernel's c2
        lib.fake_capture(b"adam_kernel", 7, 4)
        assert m.train(epochs, batch) == 0
        n = m.launches("adam_kernel")
        return m.captured(np.float32, 0)[0], m.captured(np.float32, n - 1)[0]
    assert m.train(epochs, batch) == 0
    steps = epochs * -(-rows // batch)
    c = np.ctypeslib.as_array(C.cast(lib.fake_block(8 * steps), C.POINTER(C.c_float)), (2 * steps,))
    return c[steps], c[2 * steps - 1]


@pytest.mark.parametrize("kind,rows,batch,epochs,fails,nth,done", [
    ("ta3s", 500, 100, 3, "cudaMalloc", 1, 0),                       # no room for the bias corrections
    ("ta3s", 500, 100, 3, "cudaLaunchKernel", 0, 0),                 # all 15 steps are one launch
    ("ta3s", 1, 64, 5000, "cudaLaunchKernel", 1, 4096),              # the second launch of two
    ("ta3s", 2500, 1100, 3, "cudaLaunchKernel", 6, 3),               # two launches a step
    ("ta3s", 2500, 1100, 3, "cudaLaunchKernel", 7, 3),
    ("ta3w", 500, 100, 3, "cudaMalloc", 1, 0),                       # no room for the activations
    ("ta3w", 500, 100, 3, "cudaLaunchKernelExC", 15, 2)])            # six launches a step
def test_only_steps_that_ran_count_for_the_bias_corrections(lib, kind, rows, batch, epochs, fails, nth, done):
    m = fake_cuda.Model(lib, kind)
    assert m.set_data(rows) == 0
    lib.fake_reset()
    lib.fake_fail(fails.encode(), nth)
    assert m.train(epochs, batch) == 1
    lib.fake_reset()
    steps = epochs * -(-rows // batch)
    first, last = _corrections(m, epochs, batch, rows)
    b2 = float(np.float32(0.999))
    assert abs(first - (1 - b2 ** (done + 1))) < 1e-6
    assert abs(last - (1 - b2 ** (done + steps))) < 1e-6
    m.close()


@pytest.mark.parametrize("batch", [101, 1200, 2**31 - 1, 2**31, 2**32 - 1])
def test_a_minibatch_larger_than_the_rows_is_all_rows(lib, batch):
    """Also where the argument does not fit an int, or the sum that rounds the steps up wraps around."""
    m = fake_cuda.Model(lib, "ta3s")
    assert m.set_data(100) == 0
    lib.fake_reset()
    lib.fake_capture(b"train_kernel", 0, 64)
    assert m.train(3, batch) == 0
    assert m.launches("train_kernel") == 1
    assert m.captured(np.int32)[6] == 100                            # Params: three pointers, then the batch
    assert lib.fake_block(4 * 3 * 100)                               # the shuffled rows of three epochs, no more
    m.close()


@pytest.mark.parametrize("rows,locked", [(800, 1), (262_144, 1), (262_145, 0)])
def test_page_locked_results_are_bounded(lib, rows, locked):
    """A model locks at most 2 MB of memory for its predictions; larger ones come through device memory."""
    m = fake_cuda.Model(lib, "ta3s")
    lib.fake_reset()
    assert m.predict(rows) == 0
    assert m.launches("cudaHostAlloc") == locked
    assert bool(lib.fake_block(8 * rows)) == (not locked)
    m.close()
