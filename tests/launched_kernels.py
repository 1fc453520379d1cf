"""Names of the kernels that a call launches, from a graph that it is captured into (nothing runs).  A profiler would tell them too, but
finds nothing in a process that has captured graphs since it was used last."""
import os
import tempfile

import torch


def kernels(call, names):
    """Which of `names` (a substring of the kernel's name -> what it is called here) the call launches, sorted, one entry per launch.
    It is called twice: once as it is (what it prepares on the first call stays outside the graph)."""
    call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    graph.enable_debug_mode()
    with torch.cuda.graph(graph):
        call()
    with tempfile.TemporaryDirectory() as folder:
        path = os.path.join(folder, "graph.dot")
        graph.debug_dump(path)
        with open(path) as f:
            nodes = [n for n in f.read().split("label=") if "KERNEL" in n]
    graph.reset()
    assert nodes
    return sorted(names[k] for n in nodes for k in names if k in n)
