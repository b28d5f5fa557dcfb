#!/bin/bash
# Builds libquark_b200.so (sm_100a only) next to the Python package.  Usage: build.sh [-v]
# QB_BUILD_DIR puts objects and library there instead (and leaves the extension out), with QB_BUILD_FLAGS for the compiler.
set -e
HERE="$(cd "$(dirname "$0")" && pwd)"
OUT="$HERE/../libquark_b200.so"
OBJ="$HERE/build"
if [ -n "$QB_BUILD_DIR" ]; then
  OUT="$QB_BUILD_DIR/libquark_b200.so"
  OBJ="$QB_BUILD_DIR"
fi
NVCC="${NVCC:-nvcc}"
FLAGS="-gencode arch=compute_100a,code=sm_100a -lineinfo -O3 -std=c++17 -Xcompiler -fPIC $QB_BUILD_FLAGS"
[ "$1" = "-v" ] && FLAGS="$FLAGS -Xptxas -v"
mkdir -p "$OBJ"
pids=()
for f in runtime gemm gemm_pair gemm_grouped attn attn3 kv glue qkv_post tp; do
  $NVCC $FLAGS -c "$HERE/$f.cu" -o "$OBJ/$f.o" &
  pids+=($!)
done
for p in "${pids[@]}"; do wait $p; done
$NVCC -shared -o "$OUT" "$OBJ"/{runtime,gemm,gemm_pair,gemm_grouped,attn,attn3,kv,glue,qkv_post,tp}.o -cudart static
[ -n "$QB_BUILD_DIR" ] && exit 0
# The C side of the smallest calls (a CPython extension); without the interpreter's headers they stay in Python.
PYTHON="${PYTHON:-python3}"
PYINC="$($PYTHON -c 'import sysconfig; print(sysconfig.get_paths()["include"])')"
# (named for the interpreter it was built for: another one does not import it)
EXT="$HERE/../_fastcall$($PYTHON -c 'import sysconfig; print(sysconfig.get_config_var("EXT_SUFFIX"))')"
rm -f "$EXT" "$HERE/../_fastcall.so"
if [ -f "$PYINC/Python.h" ]; then
  ${CC:-gcc} -O2 -Wall -std=gnu11 -fPIC -shared -I"$PYINC" "$HERE/fastcall.c" -o "$EXT"
else
  echo "no Python.h under $PYINC: the C side of small calls is not built"
fi
echo "built $OUT"
