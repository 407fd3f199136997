"""Nothing that clears memory may run beside the window pass of a fused call, which reports its
waits in a word that the host reads afterwards: the call is captured into a graph, and every
memset of it comes before or after the window pass along its edges."""
import re

import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("S,npix", [(3, 30), (20, 260)])  # exposure on the caller's stream; on one of its own
def test_clears_are_ordered(tmp_path, S, npix):
    import torch

    from xtsrcmaps_b200 import api as A
    from xtsrcmaps_b200.synth import make_job
    from xtsrcmaps_b200.wcs import Wcs

    A.init(0)
    d = torch.device("cuda")
    job = make_job("c1", seed=5, n_sources=S)
    t = lambda v: torch.as_tensor(np.ascontiguousarray(v), device=d)  # noqa: E731
    tg = lambda g: type(g)(t(g.cosths), t(g.logEs), t(g.params), g.min_cos_theta)  # noqa: E731
    tc = lambda c: A.ExpCube(t(c.cosbins), c.nside, c.nbrbins, c.cosmin, c.thetabin)  # noqa: E731
    w = job.wcs
    wcs = Wcs(npix, npix, (npix + 1) / 2.0, (npix + 1) / 2.0, w.crval1, w.crval2, -0.1, 0.1)
    args = (wcs, t(job.src_sph), tc(job.exp_cube), tc(job.wexp_cube), t(job.logEs), tg(job.aeff_front),
            tg(job.aeff_back), tg(A.normalize_rpsf(job.rpsf_front, job.scale_front)),
            tg(A.normalize_rpsf(job.rpsf_back, job.scale_back)),
            t(A.livetime_efficiency_factors(job.logEs, job.effic_front)))
    st = torch.cuda.Stream()
    with torch.cuda.stream(st):
        out, _ = A.point_source_maps(*args, with_info=False)
    st.synchronize()
    g = torch.cuda.CUDAGraph(keep_graph=True)  # (kept for the dump)
    g.enable_debug_mode()
    with torch.cuda.graph(g, stream=st):
        A.point_source_maps(*args, out=out, with_info=False)
    dot = tmp_path / "graph.dot"
    g.debug_dump(str(dot))
    text = dot.read_text()
    kind = dict(re.findall(r'"(graph_\d+_node_\d+)"\[.*?label="\{(\w+)', text))
    nodes = dict(re.findall(r'"(graph_\d+_node_\d+)"\[(.*?)\];\n', text, re.S))
    after = {n: set() for n in nodes}
    for a, b in re.findall(r'"(graph_\d+_node_\d+)" -> "(graph_\d+_node_\d+)"', text):
        after[a].add(b)

    def reached(n):
        seen, todo = set(), [n]
        while todo:
            for m in after[todo.pop()] - seen:
                seen.add(m)
                todo.append(m)
        return seen

    windows = [n for n, v in nodes.items() if "k_pixel_windows" in v]
    clears = [n for n in nodes if kind.get(n) == "MEMSET"]
    assert len(windows) == 1 and clears
    for c in clears:
        assert windows[0] in reached(c) or c in reached(windows[0])
    del g
