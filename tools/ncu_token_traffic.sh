#!/bin/bash
# DRAM bytes of every kernel of one decode token (cheap metric pass) → token_traffic_<model>.csv in the folder $OUT (default: here)
set -u
M=${1:-Qwen2.5-0.5B}
OUT=${OUT:-.}
timeout 600 ncu --metrics dram__bytes_read.sum,dram__bytes_write.sum,gpu__time_duration.sum --clock-control none \
  --profile-from-start off --csv --log-file $OUT/token_traffic_$M.csv python tools/profile_decode.py $M 1 > /dev/null 2>&1
wc -l $OUT/token_traffic_$M.csv
