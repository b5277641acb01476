#!/usr/bin/env bash
# Builds, in-tree, the cs2d shared library for sm_100a and the native host path of the PyTorch operators.
#   official-cross-scan_b200/csrc/build.sh [extra nvcc flags]
# CS2D_OUT=<file> writes the library elsewhere (and leaves the PyTorch module alone).
set -euo pipefail
here="$(cd "$(dirname "${BASH_SOURCE[0]}")" && pwd)"
out="${CS2D_OUT:-$here/../cs2d/libcs2d.so}"
NVCC="${NVCC:-/usr/local/cuda/bin/nvcc}"
CUDA="$(dirname "$(dirname "$NVCC")")"
PYTHON="${PYTHON:-python3}"
ti="$("$PYTHON" -c 'import os, importlib.util as u; print(os.path.dirname(u.find_spec("torch").origin))')"
tmp="$(mktemp -d)"
trap 'rm -r "$tmp"' EXIT
native=""
if [ -z "${CS2D_OUT:-}" ]; then   # host code only: compiled while nvcc runs, linked once the library is there
  g++ -O2 -std=c++17 -fPIC -fvisibility=hidden -DTORCH_EXTENSION_NAME=_native -DTORCH_API_INCLUDE_EXTENSION_H \
    -isystem "$ti/include" -isystem "$ti/include/torch/csrc/api/include" -isystem "$CUDA/include" \
    -isystem "$("$PYTHON" -c 'import sysconfig; print(sysconfig.get_paths()["include"])')" \
    -c "$here/cs2d_torch.cpp" -o "$tmp/cs2d_torch.o" & native=$!
fi
"$NVCC" -gencode arch=compute_100a,code=sm_100a -lineinfo -O3 -std=c++17 \
  -Xcompiler -fPIC,-Wformat,-Werror=format,-Werror=format-extra-args -shared -cudart static --threads 0 "$@" -Xlinker -soname=libcs2d.so \
  -o "$out" "$here/cs2d_api.cu" "$here/cs2d_fwd.cu" "$here/cs2d_bwd.cu" "$here/cs2d_fwd_serial.cu" "$here/cs2d_bwd_serial.cu" "$here/cs2d_stream_fwd.cu" "$here/cs2d_stream_bwd.cu" "$here/cs2d_walk_fwd.cu" "$here/cs2d_blk_fwd.cu" "$here/cs2d_blk_bwd.cu" "$here/cs2d_pair_fwd.cu" "$here/cs2d_pair_bwd.cu"
echo "built $out"
if [ -n "$native" ]; then
  wait "$native"
  lib="$here/../cs2d"
  g++ -shared -o "$lib/_native.so" "$tmp/cs2d_torch.o" -L"$lib" -l:libcs2d.so -L"$ti/lib" -lc10 -lc10_cuda -ltorch_cpu -ltorch \
    -ltorch_python -L"$CUDA/lib64" -lcudart_static -ldl -lrt -lpthread -Wl,-rpath,'$ORIGIN'
  echo "built $lib/_native.so"
fi
