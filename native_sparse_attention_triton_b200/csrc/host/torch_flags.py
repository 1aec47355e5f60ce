"""Prints the compiler or linker flags for an extension of the torch that this interpreter imports."""
import os
import sys
import sysconfig

import torch

root = os.path.dirname(torch.__file__)
cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
if sys.argv[1] == "compile":
    include = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"), os.path.join(cuda, "include"),
               sysconfig.get_paths()["include"]]
    print(f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", *[f"-isystem {p}" for p in include])
else:
    libs = ["c10", "c10_cuda", "torch", "torch_cpu", "torch_cuda", "torch_python"]
    print(f"-L{os.path.join(root, 'lib')} -L{os.path.join(cuda, 'lib64')}", *[f"-l{n}" for n in libs], "-lcudart")
