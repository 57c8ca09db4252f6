#!/bin/bash
# ncu --set full capture of one cluster-resident decode step (decode_stack_kernel) at the headline shape, mid context: the fifth step behind prompts of 130 tokens (position 135; 1 GB on the device).
mkdir -p gpurun_out
CMD="python scripts/ncu_headline_step.py"
$CMD > gpurun_out/ncu_stack_plain.log 2>&1 &&
ncu --set full --clock-control none -k regex:decode_stack_kernel -s 4 -c 1 -f -o gpurun_out/stack $CMD > gpurun_out/ncu_stack.log 2>&1
echo "ncu rc=$?"; tail -3 gpurun_out/ncu_stack.log
