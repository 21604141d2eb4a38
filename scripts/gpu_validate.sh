#!/usr/bin/env bash
# Validation on one B200: the GPU tests, the smoke step, the default benchmark and its reference arm.  Logs go to the folder given as the first
# argument (a temporary one without it).  Counters are taken apart from this, on one kernel of a small case at a time.
set -x
out=${1:-$(mktemp -d)}
mkdir -p "$out"
timeout 1200 python -m pytest tests -q -m gpu --timeout 300 --timeout-method=thread 2>&1 | tail -5
timeout 300 python -c "import __graft_entry__ as g; g.smoke(); print('SMOKE OK')" 2>&1 | tail -2
timeout 900 python bench.py --steps 5 --warmup 3 > "$out/bench_n1.json" 2> "$out/bench_n1.err"
python -c "
import json, sys; d=json.loads(open(sys.argv[1]).read().strip().splitlines()[-1]); print(d['ms_per_step'], d['value'], d['clocks'], d['gpu_launches'], d['roofline']['kernel'], d['roofline']['frac'], d['roofline']['traffic']); print({k:round(v['ms_per_step'],2) for k,v in d['roofline']['per_kernel'].items()}); print(d['roofline'].get('component_ms_per_step'))" "$out/bench_n1.json"
timeout 400 python bench.py --impl reference --steps 2 --warmup 1 > "$out/bench_ref.json" 2> "$out/bench_ref.err"; cut -c1-300 "$out/bench_ref.json"
