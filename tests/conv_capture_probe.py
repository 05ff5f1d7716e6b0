"""Helper of tests/test_learned_gpu.py::test_first_convolution_under_capture: the first
nn_* call of the process, a convolution, inside a stream capture; replayed, then compared
with the same call outside."""
import ctypes as C

import torch

from nga2_b200 import learned as NL

L = NL.lib()
shape, c = (1, 5, 17, 9), 32
g = torch.Generator().manual_seed(1)
x = torch.randn((5 * 17 * 9, c), generator=g).to(torch.bfloat16).cuda()
wt = (torch.randn((27, c, c), generator=g) / 30).to(torch.bfloat16).cuda()
y, z = torch.zeros_like(x), torch.zeros_like(x)


def conv(out):
    a, b = NL.Act(x.data_ptr(), *shape, c, c), NL.Act(out.data_ptr(), *shape, c, c)
    return L.nn_conv3(C.byref(a), wt.data_ptr(), None, C.byref(b), 1, torch.cuda.current_stream().cuda_stream)


graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    st = conv(y)
print("status under capture", st)
assert st == 0
graph.replay()
torch.cuda.synchronize()
assert conv(z) == 0
torch.cuda.synchronize()
assert torch.equal(y, z) and float(y.float().abs().sum()) > 0
print("capture ok")
