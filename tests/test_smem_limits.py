"""Dynamic shared-memory limits of the library's kernels.

cudaFuncAttributeMaxDynamicSharedMemorySize belongs to a kernel and a device,
so every host thread's contexts share it.  A limit set to one context's sizes
can be lowered by another thread between that context's setting and its launch,
which is then refused.  So the attribute is set in one helper only, whose value
is a compile-time constant of the kernel."""
from tests.test_stream_order import _calls, _sources


def test_limits_are_constants_of_the_kernel():
    where = []
    for f in _sources():
        text = f.read_text()
        where += [(f.name, line) for line, _ in _calls(text, "cudaFuncSetAttribute")]
    assert [w[0] for w in where] == ["common.cuh"], where
