"""Which kernels a call launches: the call is captured into a CUDA graph and the
graph's own description is searched for kernel names.  For calls that can be
captured (no allocation by the library, no wait)."""
import os
import re
import tempfile
import warnings

import torch


def launched(fn, *names):
    """The subset of `names` among the kernels that fn() launches: kernel names, with the
    first template arguments in their mangled form (I..) where these matter."""
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    graph.enable_debug_mode()
    with torch.cuda.graph(graph):
        fn()
    with tempfile.TemporaryDirectory() as d, warnings.catch_warnings():
        warnings.simplefilter("ignore")  # (it warns that it writes the file)
        path = os.path.join(d, "graph.dot")
        graph.debug_dump(path)
        text = open(path).read()
    # mangled names: length of the identifier, then the identifier
    return {n for n in names if f"{len(re.match('[a-z0-9_]+', n)[0])}{n}" in text}
