"""Which convection kernel a context runs, as it tells it: by the arithmetic, the
slice's shape and what its planes need."""
import pytest

from verb4d_b200 import Context, VerbError

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("arith,shape,kernel", [
    ("exact", (48, 101, 101, 8), "staged"), ("exact", (48, 101, 101, 91), "lines"),
    ("exact", (9, 25, 4, 4), "lines"), ("stream", (48, 101, 101, 91), "staged"),
    ("stream", (60, 150, 3, 2), "stream"), ("stream", (11, 2, 3, 2), "lines"),
    ("fma", (48, 101, 101, 8), "lines")])
def test_kernel(gpu, arith, shape, kernel):
    c = Context(*shape)
    c.set_convection_arith(arith)
    assert c.convection_kernel() == kernel
    c.close()


def test_no_kernel(gpu):
    c = Context(3, 600, 2, 2)  # lines longer than any kernel's
    with pytest.raises(VerbError):
        c.convection_kernel()
    c.close()
