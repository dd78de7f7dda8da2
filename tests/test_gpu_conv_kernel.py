"""Which convection kernel a context runs, as it tells it: by the arithmetic, the
slice's shape and what its planes need."""
import pytest

from verb4d_b200 import Context, VerbError

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("arith,shape,kernel", [
    ("exact", (48, 101, 101, 8), "staged"), ("exact", (48, 101, 101, 91), "lines"),
    ("exact", (2, 25, 4, 4), "lines"), ("stream", (48, 101, 101, 91), "staged"),
    ("stream", (60, 150, 3, 2), "stream"), ("stream", (11, 2, 3, 2), "lines"),
    ("fma", (48, 101, 101, 8), "lines")])
def test_kernel(gpu, arith, shape, kernel):
    c = Context(*shape)
    c.set_convection_arith(arith)
    assert c.convection_kernel() == kernel
    c.close()


@pytest.mark.parametrize("shape,status", [((2, 600, 2, 2), "VERB_ERR_SIZE"),  # longer than any kernel's lines
                                          ((9, 25, 2, 2), "VERB_ERR_GRID")])
def test_no_kernel(gpu, shape, status):
    c = Context(*shape)
    with pytest.raises(VerbError) as e:
        c.convection_kernel()
    c.close()
    assert status in str(e.value)
