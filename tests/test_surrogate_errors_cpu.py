"""A product whose wait ran out leaves rows unwritten and sets the network's
error flag: inference must report it, as training does."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oqupy_gb300 import _native as nat, surrogate as sg  # noqa: E402


class Net:
    """What Surrogate uses of Mlp, without a GPU."""
    torch, dev = torch, torch.device("cpu")

    def __init__(self, err):
        self.err = torch.full((1,), err, dtype=torch.int32)

    def forward(self, X):
        return torch.zeros(len(X), 6)

    check_errors = sg.Mlp.check_errors


def surrogate(err):
    s = sg.Surrogate.__new__(sg.Surrogate)
    s.net, s.nsteps, s.dt, s.residual, s.bins, s.err_map = Net(err), 2, 0.05, False, 1, np.zeros(1)
    s.lo, s.hi = (np.array([sg.BOX[k][i] for k in sg.KEYS]) for i in (0, 1))
    return s


def test_predict_reports_the_error_flag():
    P = sg.sample_params(3, 1)
    assert surrogate(0).predict(P).shape == (3, 3, 2)
    for call in (lambda s: s.predict(P), lambda s: s.screen(P), lambda s: s.calibrate(P, np.zeros((3, 3, 2)))):
        with pytest.raises(nat.DeviceError):
            call(surrogate(1))
