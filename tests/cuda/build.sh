#!/bin/bash
# Build the standalone CUDA test binaries (cross-compiles without a GPU): build.sh [output folder, default bin]
set -e
cd "$(dirname "$0")"
OUT=${1:-bin}
FLAGS="-gencode arch=compute_100a,code=sm_100a -O3 -std=c++17 -lineinfo"
mkdir -p "$OUT"
# the kernels' sources are those of the extension's build
LIST=$(python3 ../../mlx_sharding_b200/ops/build.py --gemm-sources)
mapfile -t SRC <<< "$LIST"
OBJ=()
JOBS=()
for f in "${SRC[@]}" gemm_test.cu gemm_sweep.cu; do
  nvcc $FLAGS -I ../../mlx_sharding_b200/ops/csrc -c -o "$OUT/$(basename "$f" .cu).o" "$f" &
  JOBS+=($!)
done
for j in "${JOBS[@]}"; do wait "$j"; done
for f in "${SRC[@]}"; do OBJ+=("$OUT/$(basename "$f" .cu).o"); done
for b in gemm_test gemm_sweep; do nvcc $FLAGS -o "$OUT/$b" "$OUT/$b.o" "${OBJ[@]}"; done
echo built
