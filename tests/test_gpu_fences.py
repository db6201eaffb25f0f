"""A fence covers its submission, every earlier one on the queue and those that
these waited for through semaphores: what they wrote in host-visible memory is
there for the host once the fence has been waited for, whatever fences the earlier ones had and whether those were ever
looked at, and a fence that is looked at late takes nothing back from the
host. Bytes against one array per memory."""
import ctypes

import numpy as np
import pytest

from tests.test_gpu_host_memory import DST, SIZE, SRC, BeginInfo, BufferInfo, CommandInfo, FenceInfo, MemoryInfo, SubmitInfo, Vulkan, struct, u32, u64, vp

pytestmark = pytest.mark.gpu

SemaphoreInfo = struct(u32, vp, u32)


class Submissions(Vulkan):
    """One command buffer and one fence per submission in flight."""

    def __init__(self, count=8):
        super().__init__()
        self.cmds = (vp * count)()
        info = CommandInfo(40, None, self.pool, 0, count)
        self.call("vkAllocateCommandBuffers", vp(self.device), ctypes.byref(info), self.cmds)
        self.fences = [self.make("vkCreateFence", vp(self.device), FenceInfo(8)) for _ in range(count)]

    def send(self, k, queue, record, fence=False, waits=(), signals=()):
        """Submits command buffer k, with fence k when asked."""
        self.cmd = vp(self.cmds[k])
        begin = BeginInfo(42)
        self.call("vkBeginCommandBuffer", self.cmd, ctypes.byref(begin))
        record()
        self.call("vkEndCommandBuffer", self.cmd)
        w, s, stages = (vp * max(1, len(waits)))(*waits), (vp * max(1, len(signals)))(*signals), (u32 * max(1, len(waits)))(*[0x10000] * len(waits))
        info = SubmitInfo(4, None, len(waits), ctypes.addressof(w), ctypes.addressof(stages), 1, ctypes.addressof(self.cmd), len(signals), ctypes.addressof(s))
        self.call("vkQueueSubmit", queue, u32(1), ctypes.byref(info), vp(self.fences[k]) if fence else None)

    def wait(self, k):
        f = vp(self.fences[k])
        self.call("vkWaitForFences", vp(self.device), u32(1), ctypes.byref(f), u32(1), u64(2 ** 64 - 1))

    def reset(self, k):
        f = vp(self.fences[k])
        self.call("vkResetFences", vp(self.device), u32(1), ctypes.byref(f))

    def idle(self, queue):
        self.call("vkQueueWaitIdle", queue)

    def check(self, memory, model):
        host = self.mapped(memory)
        equal = np.array_equal(host, model)
        self.unmap(memory)
        return equal


def words(value, size):
    return np.tile(np.array([value], np.uint32).view(np.uint8), size // 4)


@pytest.mark.parametrize("earlier", ["without a fence", "with a fence nobody looks at"])
@pytest.mark.parametrize("usage", [DST, SRC | DST])
@pytest.mark.parametrize("mapped_before", [False, True])
def test_a_fence_covers_the_earlier_submissions(native, earlier, usage, mapped_before):
    vk = Submissions()
    target, memory = vk.buffer(usage)
    model = np.zeros(SIZE, np.uint8)
    q = vk.queues[0]
    if mapped_before:  # the first submission after a map copies its writes back itself, later ones do not
        host = vk.mapped(memory)
        host[:] = 7
        model[:] = 7
        vk.unmap(memory)
    else:
        vk.send(3, q, lambda: vk.fill(target, 0, SIZE, 0))
    for k, (at, n, value) in enumerate([(0, 1024, 0x11111111), (1024, 1024, 0x22222222), (2048, 512, 0x33333333)]):
        vk.send(k, q, lambda: vk.fill(target, at, n, value), fence=k == 2 or earlier.startswith("with a"))
        model[at:at + n] = words(value, n)
    vk.wait(2)
    assert vk.check(memory, model)
    if usage & SRC:  # nothing stale went back to the device's side at the unmap
        other, m = vk.buffer(DST)
        vk.send(4, q, lambda: vk.copy(target, other, [(0, 0, SIZE)]), fence=True)
        vk.wait(4)
        assert vk.check(m, model)


@pytest.mark.parametrize("settled_by", ["queue", "device", "later fence"])
def test_a_fence_looked_at_late_takes_nothing_back(native, settled_by):
    vk = Submissions()
    target, memory = vk.buffer(DST)
    q = vk.queues[0]
    vk.send(0, q, lambda: vk.fill(target, 0, SIZE, 0x01010101), fence=True)
    if settled_by == "queue":
        vk.idle(q)
    elif settled_by == "device":
        vk.call("vkDeviceWaitIdle", vp(vk.device))
    else:
        vk.send(1, q, lambda: None, fence=True)
        vk.wait(1)
    host = vk.mapped(memory)
    assert np.array_equal(host, words(0x01010101, SIZE))
    host[:] = np.arange(SIZE) % 251
    model = host.copy()
    vk.unmap(memory)
    vk.wait(0)
    assert vk.check(memory, model)


@pytest.mark.parametrize("usage", [DST, SRC | DST])
@pytest.mark.parametrize("seed", [1, 2, 3, 4])
def test_random_submissions(native, seed, usage):
    """Runs of one to three submissions to spans of one memory, each with a
    fence or none, one wait that covers them all, then the host reads and
    sometimes writes; fences left behind are looked at later."""
    vk = Submissions()
    rng = np.random.default_rng(seed)
    target, memory = vk.buffer(usage)
    q = vk.queues[0]
    model = np.zeros(SIZE, np.uint8)
    vk.send(0, q, lambda: vk.fill(target, 0, SIZE, 0))
    vk.idle(q)
    for step in range(80):
        late = []
        last = int(rng.integers(1, 4))
        for k in range(last):
            a, b = sorted(int(x) * 4 for x in rng.integers(0, SIZE // 4, 2))
            n, value = b - a + 4, int(rng.integers(0, 2 ** 32))
            fence = k == last - 1 or rng.random() < 0.5
            vk.send(k, q, lambda: vk.fill(target, a, n, value), fence=fence)
            model[a:a + n] = words(value, n)
            if fence:
                late.append(k)
        how = rng.integers(0, 3)
        if how == 0:
            vk.idle(q)
        else:
            vk.wait(late.pop())
            if how == 1 and late and rng.random() < 0.5:
                vk.wait(late.pop())
        if rng.random() < 0.8:
            host = vk.mapped(memory)
            assert np.array_equal(host, model), step
            a, b = sorted(int(x) for x in rng.integers(0, SIZE, 2))
            host[a:b] = rng.integers(0, 256, b - a, dtype=np.uint8)
            model[:] = host
            for k in late:  # also while it is mapped
                if rng.random() < 0.5:
                    vk.wait(k)
            assert np.array_equal(host, model), (step, "mapped")
            vk.unmap(memory)
        for k in late:
            vk.wait(k)
        for k in range(last):
            vk.reset(k)
        assert vk.check(memory, model), (step, "late")


@pytest.mark.parametrize("mapped", ["never", "before", "all along"])
@pytest.mark.parametrize("queues", [1, 2])
def test_a_fence_covers_what_its_submission_waited_for(native, mapped, queues):
    """Queue 0 writes without a fence and signals a semaphore; a submission of
    queue 0 or 1 waits for it and has the fence. The range is large enough that
    a copy back after the semaphore would still run when the fence is
    signalled."""
    vk = Submissions()
    size = 64 << 20
    b = vk.make("vkCreateBuffer", vp(vk.device), BufferInfo(12, None, 0, size, DST, 0, 0, None))
    memory = vk.make("vkAllocateMemory", vp(vk.device), MemoryInfo(5, None, size, 0))
    vk.call("vkBindBufferMemory", vp(vk.device), vp(b), vp(memory), u64(0))
    semaphore = vk.make("vkCreateSemaphore", vp(vk.device), SemaphoreInfo(9))

    def pointer():
        p = vp()
        vk.call("vkMapMemory", vp(vk.device), vp(memory), u64(0), u64(2 ** 64 - 1), u32(0), ctypes.byref(p))
        return np.ctypeslib.as_array(ctypes.cast(p, ctypes.POINTER(ctypes.c_uint32)), (size // 4,))

    if mapped != "never":
        host = pointer()
        host[:] = 5
        if mapped == "before":
            vk.unmap(memory)
    first, second = vk.queues[0], vk.queues[queues - 1]
    for value in (0x0A0A0A0A, 0x0B0B0B0B):
        vk.send(0, first, lambda: vk.fill(b, 0, size, value), signals=[semaphore])
        vk.send(1, second, lambda: None, fence=True, waits=[semaphore])
        vk.wait(1)
        if mapped != "all along":
            host = pointer()
        assert host[-1] == value  # the last to arrive
        assert np.all(host == value)
        if mapped != "all along":
            vk.unmap(memory)
        vk.reset(1)
