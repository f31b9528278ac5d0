#!/usr/bin/env bash
# The counters of $OUT/prof_<what>.ncu-rep that profiles/ keeps, as lines of target,kernel,metric,unit,value.  Runs where the report is (no GPU needed).
set -uo pipefail
cd "$(dirname "$0")/.."
echo "target,kernel,metric,unit,value"
for what in "$@"; do
  rep=${OUT:-out}/prof_$what.ncu-rep
  [ -f "$rep" ] || { echo "missing $rep" >&2; continue; }
  ncu -i "$rep" --page raw --csv 2>/dev/null | python3 -c '
import csv, re, sys
keep = re.compile(r"gpu__time_duration.sum$|launch__(grid_size|block_size|registers_per_thread|shared_mem_per_block_dynamic|waves_per_multiprocessor)$"
                  r"|sm__pipe_tensor_cycles_active.avg.pct_of_peak_sustained_active$|sm__inst_executed_pipe_xu.avg.pct|sm__inst_issued.avg.pct"
                  r"|sm__warps_active.avg.pct|l1tex__throughput.avg.pct|lts__throughput.avg.pct|gpu__dram_throughput.avg.pct|dram__bytes_(read|write).sum$"
                  r"|smsp__average_warps_issue_stalled_(barrier|long_scoreboard|short_scoreboard|wait|math_pipe_throttle)_per_issue_active.ratio$")
head, units, *rows = csv.reader(sys.stdin)
for r in rows:
    name = re.sub(r"^void |\(.*$|mdi::|hyb::", "", r[head.index("Kernel Name")]).replace(",", ";")
    for h, u, v in zip(head, units, r):
        if keep.search(h): print(",".join((sys.argv[1], name, h, u, v.replace(",", ""))))
' "$what"
done
