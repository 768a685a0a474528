"""Compiler and linker flags for an extension of the running interpreter's torch: `python fast_flags.py compile | link`."""
import os
import sys
import sysconfig

import torch
from torch.utils import cpp_extension

if sys.argv[1] == "compile":
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    dirs = list(cpp_extension.include_paths()) + [sysconfig.get_paths()["include"], os.path.join(cuda, "include")]
    print(*(f"-isystem {d}" for d in dirs), f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}")
else:
    print(*(f"-L{d} -Wl,-rpath,{d}" for d in cpp_extension.library_paths()), "-lc10 -lc10_cuda -ltorch_cpu -ltorch -ltorch_python")
