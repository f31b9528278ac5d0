#!/usr/bin/env bash
# ncu captures of the hot kernels on small cases (one GPU; never a bench value), each after the same command has run without ncu.
# Reports land in $OUT/prof_<what>.ncu-rep; summarise_ncu.sh prints the counters that profiles/ keeps of them.
set -uo pipefail
cd "$(dirname "$0")/.."
out=${OUT:-out}
mkdir -p "$out"
for what in ${@:-decode gemm attn}; do
  n=1; skip=2
  case $what in
    decode) k="regex:stream_bulk_kernel" ;;
    decode_fp8) k="regex:stream_bulk_fp8_kernel" ;;
    gemm)   k="regex:gemm_bf16_tcgen05_pair_kernel" ;;
    grouped) k="regex:gemm_grouped_tcgen05_kernel" ;;
    attn)   k="regex:attn_decode_kernel" ;;
    attnp)  k="regex:attn_prefill_tcgen05_pingpong_kernel" ;;
    gemm_fp8) k="regex:gemm_fp8_kernel" ;;
    gemm_shared) k="regex:gemm_bf16_tcgen05_kernel" ;;
    few_rows) k="regex:few_rows_linear_kernel" ;;
    chunks) k="regex:gated_chunk"; n=3; skip=6 ;;
    capped) k="regex:prompt_attn_tc_kernel" ;;
  esac
  timeout 120 python scripts/profile_targets.py $what > "$out/plain_$what.log" 2>&1 || { echo "$what failed without ncu"; exit 1; }
  timeout 600 ncu --section SpeedOfLight --section MemoryWorkloadAnalysis --section ComputeWorkloadAnalysis --section WarpStateStats \
    --section LaunchStats --section Occupancy --metrics dram__bytes_read.sum,dram__bytes_write.sum,sm__pipe_tensor_cycles_active.avg.pct_of_peak_sustained_active \
    --clock-control none -k "$k" --launch-skip $skip --launch-count $n -f \
    -o "$out/prof_$what" python scripts/profile_targets.py $what > "$out/ncu_$what.log" 2>&1
  tail -2 "$out/ncu_$what.log"
done
