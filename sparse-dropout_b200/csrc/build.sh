#!/bin/sh
# Builds libsparsedrop.so for sm_100a and, on top of it, the torch extension sd_torch.so (host code only), both next to
# the Python package (in-tree, not installed).
set -e
here="$(cd "$(dirname "$0")" && pwd)"
out="$here/../lib"
mkdir -p "$out"
NVCC="${NVCC:-/usr/local/cuda/bin/nvcc}"
PYTHON="${PYTHON:-python3}"
cuda="$(dirname "$(dirname "$NVCC")")"
torch="$("$PYTHON" -c 'import importlib.util as u; print(u.find_spec("torch").submodule_search_locations[0])')"
pyinc="$("$PYTHON" -c 'import sysconfig; print(sysconfig.get_paths()["include"])')"
"${CXX:-g++}" -std=c++17 -O2 -g0 -fPIC -fvisibility=hidden -DTORCH_EXTENSION_NAME=sd_torch -c "$here/sd_torch.cpp" -o "$out/sd_torch.o" \
    -isystem "$torch/include" -isystem "$torch/include/torch/csrc/api/include" -isystem "$pyinc" -isystem "$cuda/include" &
torch_job=$!
"$NVCC" -std=c++17 -O3 -lineinfo -gencode arch=compute_100a,code=sm_100a -t 0 \
    -Xcompiler -fPIC -Xptxas -v --shared \
    -o "$out/libsparsedrop.so" \
    "$here/sd_api.cu" "$here/sd_plan.cu" "$here/sd_gemm.cu" "$here/sd_conv.cu" "$here/sd_norm.cu" "$here/sd_cast.cu" \
    "$here/sd_optim.cu" "$here/sd_gelu.cu" "$here/sd_selftest.cu" "$@"
wait $torch_job
"${CXX:-g++}" -shared -o "$out/sd_torch.so" "$out/sd_torch.o" -L"$out" -lsparsedrop -L"$torch/lib" -lc10 -lc10_cuda -ltorch_cpu \
    -ltorch_cuda -ltorch_python -Wl,-rpath,'$ORIGIN' -Wl,-rpath,"$torch/lib"
rm -f "$out/sd_torch.o"
