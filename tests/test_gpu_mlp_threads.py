"""The warm-start object called from several threads: its entry points exclude one another, the
ones that read or replace the parameters and the normalisation included, so every result belongs
to one whole set of parameters."""
import threading

import numpy as np
import pytest

from sph_fem_2d_cutting_gpu_gb300 import abi, setups
from sph_fem_2d_cutting_gpu_gb300.solver import Solver
from test_gpu_mlp import net_with
from test_mlp_oracle import data, random_net

pytestmark = pytest.mark.gpu


def norm_list(n):
    return np.array([*n.x_mean, *n.x_std, n.y_mean, n.y_std], np.float32)


def replace_by(m, params, norm):
    n = abi.MlpNorm()
    n.x_mean[:], n.x_std[:] = list(norm[0:4]), list(norm[4:8])
    n.y_mean, n.y_std = float(norm[8]), float(norm[9])
    m.set_params(params.astype(np.float32), n)


def test_parameters_replaced_beside_other_calls(lib):
    sets = [random_net(41), random_net(42)]
    sets[1][1][8] += 0.5
    x, t = data(3000, 43)
    whole = []
    for p, norm in sets:
        m = net_with(p, norm)
        whole.append((m.gradients(x, t), m.predict(x)))
        m.close()
    m = net_with(*sets[0])
    stop, wrong = threading.Event(), []

    def replace():
        for k in range(600):
            replace_by(m, *sets[k & 1])
        stop.set()

    def gradients():
        while not stop.is_set():
            g, loss = m.gradients(x, t)
            if not any(np.array_equal(g, w[0][0]) and loss == w[0][1] for w in whole):
                wrong.append("gradients")

    def predict():
        while not stop.is_set():
            y = m.predict(x)
            if not any(np.array_equal(y, w[1]) for w in whole):
                wrong.append("predict")

    def read():
        while not stop.is_set():
            p, norm = m.params()
            if not any(np.array_equal(p, s[0].astype(np.float32)) and np.array_equal(norm_list(norm), s[1]) for s in sets):
                wrong.append("params")

    threads = [threading.Thread(target=f) for f in (replace, gradients, predict, read)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    m.close()
    assert not wrong, {w: wrong.count(w) for w in wrong}


def stepped(m):
    """The state of a yielding lattice after a step with the object's parameters as warm start."""
    s = Solver(setups.micro(n_side=48, seed=3), abi.SPH_PREC_FP32K)
    s.attach_mlp(m)
    s.step(1)
    out = s.download(["eps_pl", "eps_pl_dot", "S"])
    s.close()
    return out


def test_attached_beside_replacement(lib):
    """A context takes one whole set of parameters: it steps as with the one or with the other."""
    sets = [random_net(44), random_net(45)]
    whole = []
    for p, norm in sets:
        m = net_with(p, norm)
        whole.append(stepped(m))
        m.close()
    assert not np.array_equal(whole[0]["eps_pl_dot"], whole[1]["eps_pl_dot"])
    m = net_with(*sets[0])
    stop = threading.Event()

    def replace():
        k = 0
        while not stop.is_set():
            k += 1
            replace_by(m, *sets[k & 1])

    th = threading.Thread(target=replace)
    th.start()
    try:
        got = [stepped(m) for _ in range(40)]
    finally:
        stop.set()
        th.join()
    m.close()
    for g in got:
        assert any(all(np.array_equal(g[f], w[f], equal_nan=True) for f in w) for w in whole)
