"""bench_out/parity_report.jsonl (every check_close / report_rel of a `pytest -m gpu` run) ->
profiles/r02_parity.md + .jsonl.  Usage: python tools/parity_table.py [jsonl]"""
import json
import sys
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent
src = Path(sys.argv[1] if len(sys.argv) > 1 else ROOT / "bench_out/parity_report.jsonl")
rows = [json.loads(l) for l in src.read_text().splitlines() if l.strip()]
seen, uniq = set(), []
for r in rows:
    if r["name"] not in seen:
        seen.add(r["name"])
        uniq.append(r)
a = [r for r in uniq if "ref_err" in r]
b = [r for r in uniq if "ref_err" not in r]
out = ["# Parity report (B200, `pytest -m gpu`), round 2", "",
       "`err` = max |CUDA - fp32 truth|; `ref err` = max |reference's own bf16 path - fp32 truth| (the oracle evaluated",
       "in bf16 with the reference's unfused rounding points; for the full-size `cfg*` rows both oracle evaluations run on",
       "the device with torch's library kernels, TF32 off); ratio 1.0 = as close to the truth as the reference itself.", "",
       "| check | max abs truth | err | rel err | ref err | ratio (max) | ratio (rms) | bound factor |", "|---|---|---|---|---|---|---|---|"]
for r in a:
    out.append("| %s | %.3f | %.3e | %.2e | %.3e | **%.2f** | %.2f | %.2g |" % (
        r["name"], r["scale"], r["err"], r["rel_err"], r["ref_err"], r["ratio_max"], r["ratio_rms"], r.get("factor", 2)))
out += ["", "Kernel-level checks against fp32 math on bf16-rounded inputs (`rel err` = max abs error / max |ref|):", "",
        "| check | max abs ref | rel err | rms err | tolerance |", "|---|---|---|---|---|"]
for r in b:
    out.append("| %s | %.3f | %.2e | %.2e | %s |" % (r["name"], r["scale"], r["rel_err"], r["rms_err"],
                                                    "%.1e" % r["tol"] if "tol" in r else "2^-7 + 1e-3"))
(ROOT / "profiles/r02_parity.md").write_text("\n".join(out) + "\n")
(ROOT / "profiles/r02_parity_report.jsonl").write_text("\n".join(json.dumps(r) for r in uniq) + "\n")
print("\n".join(out[:40]))
