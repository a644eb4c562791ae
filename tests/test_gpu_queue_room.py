"""The interface queue's room: pgdg_tune("iface_cap", -1) after a fixed capacity, and a
queue switched off after it grew, batch a stage's problems again as an untouched
context does."""
import pytest

pytestmark = pytest.mark.gpu


def _batched(g):
    """Problems the last stage solved as a batch."""
    g.sync()
    g.set_iface_queue(True)
    n = len(g.iface_problems()[0])
    g.set_iface_queue(False)
    return n


@pytest.mark.parametrize("prec", [1, 2])
@pytest.mark.parametrize("how", ["off", "queued", "network"])
def test_automatic_room_returns(gpu_mod, prec, how):
    """Capacity 1, then automatic again: with the queue off all along, while it is on,
    and while a network is attached that is taken off again."""
    M = gpu_mod
    from pgdg_p2_gb300 import surrogate as S
    cs, p, c = M.make_case(3, (48, 12, 12))
    n = []
    for fixed in (False, True):
        g = M.MPM(cs, prec)
        g.upload_particles(p)
        g.upload_cells(c)
        net = S.Surrogate(S.load_default()) if how == "network" else None
        if fixed:
            if how == "queued":
                g.set_iface_queue(True)
            if net:
                g.set_surrogate(net)
            g.tune("iface_cap", 1)
            g.tune("iface_cap", -1)
            if net:
                g.set_surrogate(None)
            g.set_iface_queue(False)
        g.advance(1)
        n.append(_batched(g))
        g.close()
        if net:
            net.close()
    assert n[0] > 1 and n[1] == n[0]


def test_resized_queue_holds_no_problems(gpu_mod):
    """The last stage's problems go with the buffers that held them."""
    M = gpu_mod
    cs, p, c = M.make_case(3, (48, 12, 12))
    g = M.MPM(cs, 1)
    g.upload_particles(p)
    g.upload_cells(c)
    g.set_iface_queue(True)
    g.advance(1)
    g.sync()
    assert len(g.iface_problems()[0]) > 1
    g.tune("iface_cap", 1)
    assert len(g.iface_problems()[0]) == 0
    g.tune("iface_cap", -1)
    g.advance(1)
    g.sync()
    assert len(g.iface_problems()[0]) > 1
    g.close()
