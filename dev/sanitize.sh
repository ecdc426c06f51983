#!/usr/bin/env bash
# One compute-sanitizer pass over named native kernels (needs a B200 where the tool may run).
#   bash dev/sanitize.sh memcheck|racecheck|initcheck NAME[,NAME...]
# Runs the cases of tests/gpu_kernel_check.py (kernels against their fp32 references, --quick sizes) whose names begin with one of
# NAME; racecheck looks at the shared-memory pipelines, memcheck and initcheck at global memory.  Expect a 10-50x slowdown, so one tool and few cases at a
# time.  synccheck is not offered: it aborts the launch at mbarriers whose last phase nobody waits for, which is how the pipelines end.
set -euo pipefail
TOOL=${1:?tool}
ONLY=${2:?names of kernel checks}
case "$TOOL" in memcheck|racecheck|initcheck) ;; *) echo "unknown tool: $TOOL" >&2; exit 2 ;; esac
OUT=sanitize_out
mkdir -p "$OUT"
python tests/gpu_kernel_check.py --quick --only "$ONLY" --out "$OUT/plain.json"
status=0
timeout 1500 compute-sanitizer --tool "$TOOL" --error-exitcode 9 --print-limit 20 \
  python tests/gpu_kernel_check.py --quick --only "$ONLY" --out "$OUT/$TOOL.json" > "$OUT/$TOOL.log" 2>&1 || status=$?
grep -E "ERROR SUMMARY|RACECHECK SUMMARY|Error:|Hazard" "$OUT/$TOOL.log" | head -20 || true
exit $status
