"""Linear system operator, easier/numeric/linsys.py:10-24."""
from torch import nn

from .. import ops


class Linsys(nn.Module):
    """``A(x) = reducer(selector(x) * Ae) + x * Av``.

    A call runs the product as one kernel over the Selector's index and the
    Reducer's segments, bitwise the five operations (``ops.linsys_apply``;
    anything it does not cover runs them one by one); the fused solvers turn
    the Linsys into a SELL-32 matrix (``sparse.py``) once.
    """

    def __init__(self, Av, Ae, selector, reducer) -> None:
        super().__init__()
        self.Av = Av
        self.Ae = Ae
        self.selector = selector
        self.reducer = reducer

    def forward(self, x):
        y = ops.linsys_apply(self, x)
        return y if y is not None else self.reducer(self.selector(x) * self.Ae) + x * self.Av
