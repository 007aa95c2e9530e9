"""Publication of the partial sums inside the cooperative BiCGStab launch.  A
relaxed store makes earlier stores of the block visible to its reader only if
the same thread has fenced before it; results cannot show a missing fence, so
the code is read: every store of a partial is guarded by the condition of a
fence before it in the same function, and every poll is an acquire."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = open(os.path.join(ROOT, "xamg-test_b200", "csrc", "kernels.cu")).read()


def body(name):
    a = SRC.index("auto %s = [&]" % name)
    return SRC[a:SRC.index("\n    };", a)]


def test_the_publishing_threads_fence():
    b = body("publish")
    fence = re.findall(r"if \(([^;]*?)\) grid_fence\(\);", b)
    put = re.findall(r"if \(([^;]*?)\) slot_put\(", b)
    assert len(fence) == len(put) == 1 and b.count("grid_fence()") == b.count("slot_put(") == 1
    assert fence == put and b.index("grid_fence()") < b.index("slot_put(")
    assert b.index("__syncthreads()") < b.index("grid_fence()")  # behind the block's vector stores


def test_the_meeting_thread_fences():
    b = body("meet")
    assert re.search(r"if \(wl == 0\) \{\s*grid_fence\(\);\s*slot_put\([^;]*;\s*\}", b)


def test_fence_and_polls():
    assert 'grid_fence() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }' in SRC
    get = SRC[SRC.index("bool slot_get("):]
    assert "ld.acquire.gpu.global.v2.u64" in get[:get.index("\n}")]
