"""i2g_get_markers_dev and i2g_get_nodes_dev against the host read-out of the same
context (copies: bitwise).  Marker counts below and above the size where an
unrelated caller order takes the staged form (96 MB of outputs), not multiples of
its bands of 2048 indices; every field or some; arrays aligned to 16 or only to 8
bytes; arrays that overlap, which cudaMemcpy serves as before."""
import ctypes as C

import numpy as np
import pytest

from i2elvis_planet_b200 import abi, lib, synth

pytestmark = pytest.mark.gpu

FIELDS = ("x", "y", "T", "eta", "p")


def context(n, k, count, order, precision=abi.PREC_MIXED):
    inst = synth.make_instance("r", n=n, k=k, nsteps=1, seed=5)
    idx = np.arange(inst.marknum)
    if order == "random":
        idx = np.argsort(synth.rng_u64(3, 1, inst.marknum), kind="stable")
    ms = lib.MarkerStep.from_instance(synth.subset(inst, idx[:count]), precision=precision)
    ms.movemark(inst.timestep, inst.timesum)
    ms.ronurecalc(inst.timesum)
    return ms


def read(ms, fields, offset):
    import torch
    n, nn = ms.n, ms.nodenum
    mk = {f: torch.full((n + offset,), -7.0, dtype=torch.float64, device="cuda") for f in fields}
    nd = {f: torch.full((nn + offset,), -7.0, dtype=torch.float64, device="cuda") for f in synth.NODE_OUT}
    torch.cuda.synchronize()
    p = lambda t: C.c_void_p(t.data_ptr() + 8 * offset)  # noqa: E731
    ms._check(ms.lib.i2g_get_markers_dev(ms.h, n, *[p(mk[f]) if f in mk else None for f in FIELDS]), "markers")
    ms._check(ms.lib.i2g_get_nodes_dev(ms.h, *[p(nd[f]) for f in synth.NODE_OUT]), "nodes")
    for d in (mk, nd):
        for t in d.values():
            assert (t[:offset] == -7.0).all()
    return ({f: t[offset:].cpu().numpy() for f, t in mk.items()}, {f: t[offset:].cpu().numpy() for f, t in nd.items()})


@pytest.mark.parametrize("n,k,count,order", [(21, 3, 1, "cell"), (22, 4, 2047, "random"), (401, 4, 2559999, "random"),
                                             (401, 4, 2550785, "cell"), (421, 6, 6245377, "random")])
def test_device_readout_equals_host(n, k, count, order):
    ms = context(n, k, count, order)
    mk, nodes = ms.get_markers(fields=FIELDS), ms.get_nodes()
    for fields, offset in ((FIELDS, 0), (FIELDS, 1), (("x", "eta", "p"), 0), (("T",), 1)):
        dm, dn = read(ms, fields, offset)
        for f in fields:
            np.testing.assert_array_equal(dm[f], mk[f], err_msg=f)
        for f in synth.NODE_OUT:
            np.testing.assert_array_equal(dn[f], nodes[f], err_msg=f)
    ms.step(1e12, 1e13, 2)  # the scratch the read-out used is not state
    ms.close()


def test_staged_readout_fp64_and_overlap():
    import torch
    ms = context(401, 4, 2559999, "random", abi.PREC_FP64)
    mk = ms.get_markers(fields=FIELDS)
    dm, _ = read(ms, FIELDS, 0)
    for f in FIELDS:
        np.testing.assert_array_equal(dm[f], mk[f], err_msg=f)
    # x and y into arrays that share all but one element: the copy of y comes last
    t = torch.zeros(ms.n + 1, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    ms._check(ms.lib.i2g_get_markers_dev(ms.h, ms.n, C.c_void_p(t.data_ptr()), C.c_void_p(t.data_ptr() + 8), None, None,
                                         None), "overlap")
    np.testing.assert_array_equal(t[1:].cpu().numpy(), mk["y"])
    assert float(t[0]) == mk["x"][0]
    ms.close()
