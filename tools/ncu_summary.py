#!/usr/bin/env python
"""Summarise ncu outputs into small tracked files under profiles/.

  python tools/ncu_summary.py launches launches.csv profiles/launches.md
  python tools/ncu_summary.py full prof_gemv.ncu-rep profiles/gemv_full.md
"""
import collections
import csv
import re
import subprocess
import sys

FULL_KEYS = [
    "gpu__time_duration.sum", "dram__bytes_read.sum", "dram__bytes_write.sum",
    "gpu__dram_throughput.avg.pct_of_peak_sustained_elapsed",
    "dram__cycles_active.avg.pct_of_peak_sustained_elapsed",
    "sm__throughput.avg.pct_of_peak_sustained_elapsed",
    "sm__warps_active.avg.pct_of_peak_sustained_active",
    "sm__pipe_tensor_cycles_active.avg.pct_of_peak_sustained_active",
    "sm__inst_executed_pipe_tensor.sum",
    "launch__registers_per_thread", "launch__grid_size", "launch__block_size",
    "launch__shared_mem_per_block_dynamic", "lts__t_bytes.sum",
    "l1tex__data_bank_conflicts_pipe_lsu_mem_shared.sum",
]


def launches(src, dst):
    lines = [l for l in open(src) if not l.startswith("==")]
    agg = collections.OrderedDict()
    total = 0.0
    for row in csv.DictReader(lines):
        if row.get("Metric Name") != "gpu__time_duration.sum":
            continue
        name = re.sub(r"\(.*", "", row["Kernel Name"]).replace("void ", "")
        v = float(row["Metric Value"].replace(",", ""))
        v = {"ns": v / 1e3, "us": v, "ms": v * 1e3}.get(row["Metric Unit"], v)
        key = (name, row["Grid Size"], row["Block Size"])
        agg.setdefault(key, []).append(v)
        total += v
    with open(dst, "w") as f:
        f.write(f"ncu --metrics gpu__time_duration.sum --clock-control none (cold-cache, serialised)\n\n")
        f.write("| kernel | grid | block | launches | avg us | min us | max us | total ms | share |\n"
                "|---|---|---|---|---|---|---|---|---|\n")
        for (name, g, b), v in sorted(agg.items(), key=lambda kv: -sum(kv[1])):
            f.write(f"| `{name}` | {g} | {b} | {len(v)} | {sum(v)/len(v):.2f} | {min(v):.2f} | {max(v):.2f} | "
                    f"{sum(v)/1e3:.3f} | {100*sum(v)/total:.1f}% |\n")
    print(open(dst).read())


def full(src, dst):
    out = subprocess.run(["ncu", "-i", src, "--page", "raw", "--csv"], capture_output=True, text=True).stdout
    rows = list(csv.reader(out.splitlines()))
    hdr, units = rows[0], rows[1]
    with open(dst, "w") as f:
        f.write(f"ncu --set full --clock-control none\n\n")
        for r in rows[2:]:
            f.write(f"### `{r[hdr.index('Kernel Name')]}`\n\n| metric | value | unit |\n|---|---|---|\n")
            for k in FULL_KEYS:
                if k in hdr:
                    f.write(f"| {k} | {r[hdr.index(k)]} | {units[hdr.index(k)]} |\n")
            f.write("\n")
    print(open(dst).read())


if __name__ == "__main__":
    {"launches": launches, "full": full}[sys.argv[1]](sys.argv[2], sys.argv[3])
