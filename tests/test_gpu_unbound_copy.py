"""A copy between an image and a buffer one of which has no memory is an error
of the submission, with and without gaps between the buffer's rows."""
import ctypes

import pytest

from tests.test_gpu_fences import Submissions
from tests.test_gpu_host_memory import DST, SIZE, SRC, BeginInfo, BufferInfo, MemoryInfo, SubmitInfo, struct, u32, u64, vp

pytestmark = pytest.mark.gpu

ImageInfo = struct(u32, vp, *[u32] * 11, u32, vp, u32)
Region = struct(u64, *[u32] * 12)
DEVICE_LOST = -4


@pytest.mark.parametrize("row", [0, 24])
@pytest.mark.parametrize("bound", ["image", "buffer"])
@pytest.mark.parametrize("name", ["vkCmdCopyImageToBuffer", "vkCmdCopyBufferToImage"])
def test_unbound(native, row, bound, name):
    vk = Submissions()
    # 2D RGBA8, 16 x 16 texels, one level and layer
    image = vk.make("vkCreateImage", vp(vk.device), ImageInfo(14, None, 0, 1, 37, 16, 16, 1, 1, 1, 1, 0, SRC | DST, 0, None, 0))
    if bound == "image":
        memory = vk.make("vkAllocateMemory", vp(vk.device), MemoryInfo(5, None, SIZE, 0))
        vk.call("vkBindImageMemory", vp(vk.device), vp(image), vp(memory), u64(0))
        buffer = vk.make("vkCreateBuffer", vp(vk.device), BufferInfo(12, None, 0, SIZE, SRC | DST, 0, 0, None))
    else:
        buffer, _ = vk.buffer(SRC | DST)
    region = Region(0, row, 0, 1, 0, 0, 1, 0, 0, 0, 16, 16, 1)
    cmd, begin = vp(vk.cmds[0]), BeginInfo(42)
    vk.call("vkBeginCommandBuffer", cmd, ctypes.byref(begin))
    if name == "vkCmdCopyImageToBuffer":
        vk.call(name, cmd, vp(image), u32(6), vp(buffer), u32(1), ctypes.byref(region), check=False)
    else:
        vk.call(name, cmd, vp(buffer), vp(image), u32(7), u32(1), ctypes.byref(region), check=False)
    vk.call("vkEndCommandBuffer", cmd)
    info = SubmitInfo(4, None, 0, None, None, 1, ctypes.addressof(cmd), 0, None)
    assert vk.call("vkQueueSubmit", vk.queues[0], u32(1), ctypes.byref(info), None, check=False) == DEVICE_LOST
    # the queue goes on
    other, m = vk.buffer(DST)
    vk.send(1, vk.queues[0], lambda: vk.fill(other, 0, SIZE, 0x05050505), fence=True)
    vk.wait(1)
    assert (vk.mapped(m) == 5).all()
