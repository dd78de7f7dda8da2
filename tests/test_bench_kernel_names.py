"""The benchmark names the convection kernel that its dispatch took and gives a
profiled pipe share only for the slice shape that was profiled."""
import bench


def test_named_by_the_dispatch():
    lines, share = bench.conv_kernel_entry("exact", "lines", 48, 101)
    staged, share2 = bench.conv_kernel_entry("exact", "staged", 48, 101)
    assert lines != staged and share != share2
    assert bench.conv_kernel_entry("stream", "staged", 60, 150)[1] is None
    for arith in ("exact", "fma", "stream"):
        for kernel in ("lines", "staged", "stream"):
            possible = {"exact": ("lines", "staged"), "fma": ("lines",),
                        "stream": ("lines", "staged", "stream")}[arith]
            assert ((arith, kernel) in bench.CONV_KERNEL) == (kernel in possible)
