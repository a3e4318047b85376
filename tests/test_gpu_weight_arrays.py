"""Transform weights in every form numpy turns into float64: byte orders, other
number types, lists, read-only, strided and Fortran-ordered arrays. The weights
are exact in each type, so the results are equal to the bit."""
import numpy as np
import pytest

torch = pytest.importorskip('torch')
pytestmark = pytest.mark.gpu

from mbptcode_b200 import gw, space_time                            # noqa: E402

W = np.arange(-6.0, 6.0).reshape(3, 4)


def _read_only(a):
    a = a.copy()
    a.flags.writeable = False
    return a


FORMS = {
    'big-endian': lambda a: a.astype('>f8'), 'longdouble': lambda a: a.astype(np.longdouble),
    'object': lambda a: a.astype(object), 'float32': lambda a: a.astype(np.float32),
    'int': lambda a: a.astype(np.int32), 'list': lambda a: a.tolist(), 'read-only': _read_only,
    'strided': lambda a: np.repeat(a, 2, axis=1)[:, ::2], 'Fortran': np.asfortranarray,
    'reversed': lambda a: np.ascontiguousarray(a[::-1])[::-1],
    'broadcast': lambda a: np.broadcast_to(a, (1,) + a.shape)[0]}


@pytest.mark.parametrize('form', sorted(FORMS))
def test_weights(form):
    w = FORMS[form](W)
    values = torch.arange(4 * 25, device='cuda', dtype=torch.float64).reshape(4, 5, 5)
    assert torch.equal(space_time.transform(values, w), space_time.transform(values, W))
    branch = torch.arange(2 * 4 * 7, device='cuda', dtype=torch.float64).reshape(2, 4, 7)
    assert torch.equal(gw.sigma_frequency(branch, w, w), gw.sigma_frequency(branch, W, W))
