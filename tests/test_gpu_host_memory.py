"""Coherence of host-visible memory: random sequences of host writes through
vkMapMemory, device fills and copies, submissions with and without fences,
and reads on both sides, against one array of bytes per memory. One memory
holds a buffer that the device only writes (its mirror is not uploaded at
unmap) until, in the second half, a copy reads that buffer all the same or a
second buffer that may be read is bound to the memory."""
import ctypes

import numpy as np
import pytest

import cpvulkan_gb300 as c

pytestmark = pytest.mark.gpu
u32, u64, vp = ctypes.c_uint32, ctypes.c_uint64, ctypes.c_void_p
SIZE = 4096
SRC, DST = 1, 2


def struct(*fields):
    return type("S", (ctypes.Structure,), {"_fields_": [("f%d" % i, t) for i, t in enumerate(fields)]})


InstanceInfo = struct(u32, vp, u32, vp, u32, vp, u32, vp)
QueueInfo = struct(u32, vp, u32, u32, u32, vp)
DeviceInfo = struct(u32, vp, u32, u32, vp, u32, vp, u32, vp, vp)
BufferInfo = struct(u32, vp, u32, u64, u32, u32, u32, vp)
MemoryInfo = struct(u32, vp, u64, u32)
PoolInfo = struct(u32, vp, u32, u32)
CommandInfo = struct(u32, vp, vp, u32, u32)
BeginInfo = struct(u32, vp, u32, vp)
SubmitInfo = struct(u32, vp, u32, vp, vp, u32, vp, u32, vp)
FenceInfo = struct(u32, vp, u32)
Copy = struct(u64, u64, u64)


class Vulkan:
    def __init__(self):
        lib = ctypes.CDLL(c.ICD_PATH)
        lib.vk_icdGetInstanceProcAddr.restype = vp
        lib.vk_icdGetInstanceProcAddr.argtypes = [vp, ctypes.c_char_p]
        self.lib, self.instance = lib, None
        self.instance = self.make("vkCreateInstance", None, InstanceInfo(1), device=False)
        n, pd = u32(1), vp()
        self.call("vkEnumeratePhysicalDevices", vp(self.instance), ctypes.byref(n), ctypes.byref(pd))
        priority = ctypes.c_float(1.0)
        q = QueueInfo(2, None, 0, 0, 2, ctypes.addressof(priority))
        self.device = self.make("vkCreateDevice", pd, DeviceInfo(3, None, 0, 1, ctypes.addressof(q)))
        self.queues = []
        for i in range(2):
            h = vp()
            self.call("vkGetDeviceQueue", vp(self.device), u32(0), u32(i), ctypes.byref(h), check=False)
            self.queues.append(h)
        self.pool = self.make("vkCreateCommandPool", vp(self.device), PoolInfo(39, None, 2, 0))
        self.cmd = vp()
        info = CommandInfo(40, None, self.pool, 0, 1)
        self.call("vkAllocateCommandBuffers", vp(self.device), ctypes.byref(info), ctypes.byref(self.cmd))
        self.fence = self.make("vkCreateFence", vp(self.device), FenceInfo(8))

    def call(self, name, *args, check=True):
        f = ctypes.CFUNCTYPE(ctypes.c_int)(self.lib.vk_icdGetInstanceProcAddr(self.instance, name.encode()))
        f.argtypes = None
        r = f(*args)
        assert not check or r == 0, (name, r)
        return r

    def make(self, name, parent, info, device=True):
        h = vp()
        args = ([parent] if device else []) + [ctypes.byref(info), None, ctypes.byref(h)]
        self.call(name, *args)
        return h.value

    def buffer(self, usage, memory=None):
        b = self.make("vkCreateBuffer", vp(self.device), BufferInfo(12, None, 0, SIZE, usage, 0, 0, None))
        m = memory or self.make("vkAllocateMemory", vp(self.device), MemoryInfo(5, None, SIZE, 0))
        self.call("vkBindBufferMemory", vp(self.device), vp(b), vp(m), u64(0))
        return b, m

    def submit(self, record, queue, wait):
        begin = BeginInfo(42)
        self.call("vkBeginCommandBuffer", self.cmd, ctypes.byref(begin))
        record()
        self.call("vkEndCommandBuffer", self.cmd)
        info = SubmitInfo(4, None, 0, None, None, 1, ctypes.addressof(self.cmd), 0, None)
        self.call("vkQueueSubmit", queue, u32(1), ctypes.byref(info), vp(self.fence) if wait == "fence" else None)
        if wait == "fence":
            f = vp(self.fence)
            self.call("vkWaitForFences", vp(self.device), u32(1), ctypes.byref(f), u32(1), u64(2 ** 64 - 1))
            self.call("vkResetFences", vp(self.device), u32(1), ctypes.byref(f))
        elif wait == "queue":
            self.call("vkQueueWaitIdle", queue)
        else:
            self.call("vkDeviceWaitIdle", vp(self.device))

    def fill(self, buffer, at, size, value):
        self.call("vkCmdFillBuffer", self.cmd, vp(buffer), u64(at), u64(size), u32(value), check=False)

    def copy(self, src, dst, regions):
        arr = (Copy * len(regions))(*[Copy(*r) for r in regions])
        self.call("vkCmdCopyBuffer", self.cmd, vp(src), vp(dst), u32(len(regions)), arr, check=False)

    def mapped(self, memory):
        p = vp()
        self.call("vkMapMemory", vp(self.device), vp(memory), u64(0), u64(2 ** 64 - 1), u32(0), ctypes.byref(p))
        return np.ctypeslib.as_array(ctypes.cast(p, ctypes.POINTER(ctypes.c_uint8)), (SIZE,))

    def unmap(self, memory):
        self.call("vkUnmapMemory", vp(self.device), vp(memory), check=False)


@pytest.mark.parametrize("late", ["bind", "copy"])
@pytest.mark.parametrize("seed", [1, 2, 3])
def test_random_sequences(native, seed, late):
    vk = Vulkan()
    rng = np.random.default_rng(seed)
    target, mt = vk.buffer(DST)         # the device only writes it, at first
    other, mo = vk.buffer(SRC | DST)
    memory, model = {"t": mt, "o": mo}, {}
    for k, m in memory.items():
        host = vk.mapped(m)
        host[:] = rng.integers(0, 256, SIZE, dtype=np.uint8)
        model[k] = host.copy()
        vk.unmap(m)
    readable = None

    def span():
        a, b = sorted(int(x) * 4 for x in rng.integers(0, SIZE // 4 + 1, 2))
        return a, max(b - a, 4) if a < SIZE else 4

    for step in range(160):
        if step == 80:
            readable = vk.buffer(SRC | DST, mt)[0] if late == "bind" else target
        op = rng.integers(0, 7 if readable else 5)
        queue, wait = vk.queues[rng.integers(0, 2)], ("fence", "queue", "device")[rng.integers(0, 3)]
        k = "t" if rng.random() < 0.7 else "o"
        a, n = span()
        a = min(a, SIZE - n)
        if op == 0:      # the host reads everything and writes a span
            host = vk.mapped(memory[k])
            assert np.array_equal(host, model[k]), (step, k)
            host[a:a + n] = rng.integers(0, 256, n, dtype=np.uint8)
            model[k] = host.copy()
            if rng.random() < 0.3:  # the device writes it while it is mapped
                b, m = span()
                b = min(b, SIZE - m)
                vk.submit(lambda: vk.fill(target if k == "t" else other, b, m, 0x01020304), queue, wait)
                model[k][b:b + m] = np.tile(np.array([4, 3, 2, 1], np.uint8), m // 4)
                assert np.array_equal(host, model[k]), (step, k, "mapped")
            vk.unmap(memory[k])
        elif op == 1:    # the host only reads
            host = vk.mapped(memory[k])
            assert np.array_equal(host, model[k]), (step, k)
            vk.unmap(memory[k])
        elif op == 2:
            value = int(rng.integers(0, 2 ** 32))
            vk.submit(lambda: vk.fill(target if k == "t" else other, a, n, value), queue, wait)
            model[k][a:a + n] = np.tile(np.array([value], np.uint32).view(np.uint8), n // 4)
        elif op in (3, 4):  # two separate regions from the other buffer
            half = max(4, n // 8 * 4)
            regions = [(0, a, min(half, SIZE - a)), (SIZE - 64, 0, 64)]
            vk.submit(lambda: vk.copy(other, target, regions), queue, wait)
            for s, d, m in regions:
                model["t"][d:d + m] = model["o"][s:s + m]
        else:            # the device writes and then reads the memory in one submission
            vk.submit(lambda: (vk.fill(target, a, n, 0x55AA00FF), vk.copy(readable, other, [(0, 0, SIZE)])), queue, wait)
            model["t"][a:a + n] = np.tile(np.array([0xFF, 0x00, 0xAA, 0x55], np.uint8), n // 4)
            model["o"][:] = model["t"]
    for k, m in memory.items():
        assert np.array_equal(vk.mapped(m), model[k])
        vk.unmap(m)
