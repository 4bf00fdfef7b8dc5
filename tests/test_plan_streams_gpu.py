"""A plan's tables built on one stream and read on another."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _busy(dev):
    """A stream that stays busy for some milliseconds."""
    s = torch.cuda.Stream(dev)
    with torch.cuda.stream(s):
        torch.cuda._sleep(20_000_000)
    return s


@pytest.mark.parametrize('what', ['plan', 'coarse_fft_tables', 'rows_consts', 'synth_consts', 'tc_constants'])
def test_tables_of_another_stream(what):
    from opticalimaging_b200 import engine as eng
    dev, band = torch.device('cuda', torch.cuda.current_device()), eng.Band(-29, 59, -29, 59)
    tables = {'plan': lambda p: (p.wx, p.gr, p.wn_y, p.wm_c), 'coarse_fft_tables': lambda p: p.coarse_fft_tables(),
              'rows_consts': lambda p: (p.rows_consts(0), p.rows_consts(1), p.rows_consts(2)),
              'synth_consts': lambda p: (p.synth_consts(),), 'tc_constants': lambda p: (p.tc_constants(),)}[what]
    want = tables(eng.Plan(512, 512, band, dev))
    torch.cuda.synchronize()
    plan = None if what == 'plan' else eng.Plan(512, 512, band, dev)
    with torch.cuda.stream(_busy(dev)):
        if plan is None:
            plan = eng.Plan(512, 512, band, dev)
        got = tables(plan)
    with torch.cuda.stream(torch.cuda.Stream(dev)):
        copies = [t.clone() for t in got]
    torch.cuda.synchronize()
    for c, w in zip(copies, want):
        assert torch.equal(c, w)


def test_plan_built_while_another_thread_captures():
    """The wait for a plan's tables does not break a capture (of the mode that forbids other threads to wait)."""
    import threading
    from opticalimaging_b200 import engine as eng
    dev, band = torch.device('cuda', torch.cuda.current_device()), eng.Band(-29, 59, -29, 59)
    eng.Plan(512, 512, band, dev)        # its memory stays with the allocator
    torch.cuda.synchronize()
    x, built = torch.ones(1000, device=dev), []
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode='global'):
        y = x * 2.0
        t = threading.Thread(target=lambda: built.append(eng.Plan(512, 512, band, dev)))
        t.start()
        t.join()
    graph.replay()
    torch.cuda.synchronize()
    assert len(built) == 1 and float(y[0]) == 2.0


def test_tables_built_inside_a_capture():
    from opticalimaging_b200 import engine as eng
    dev, band = torch.device('cuda', torch.cuda.current_device()), eng.Band(-29, 59, -29, 59)
    want = eng.Plan(512, 512, band, dev).coarse_fft_tables()
    plan = eng.Plan(512, 512, band, dev)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = [t.clone() for t in plan.coarse_fft_tables()]
    graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(g, w) for g, w in zip(got, want))
