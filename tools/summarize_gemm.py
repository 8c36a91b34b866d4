"""bench_out/bench_gemm.json -> profiles/r02_gemm_configs.md (markdown table)."""
import json, sys
from pathlib import Path
d = json.loads(Path(sys.argv[1] if len(sys.argv) > 1 else "bench_out/bench_gemm.json").read_text())
cfgs = ["None", "2128", "2256", "4128", "4256", "5128", "3000", "3001"]
names = {"None": "dispatch", "2128": "1-CTA 128x128", "2256": "1-CTA 128x256", "4128": "pair 256x128",
         "4256": "pair 256x256", "5128": "split-K pair", "3000": "skinny", "3001": "skinny pair"}
shapes = {
    "vit_qkv": (1024, 3456, 1152), "vit_out": (1024, 1152, 1152), "vit_fc1": (1024, 4304, 1152),
    "vit_fc2": (1024, 1152, 4304), "llm_qkv": (279, 4608, 3584), "llm_o": (279, 3584, 3584),
    "llm_gu": (279, 37888, 3584), "llm_down": (279, 3584, 18944), "proj1": (256, 3584, 4608),
    "big": (8192, 8192, 8192), "mid_vit16_qkv": (16384, 3456, 1152), "mid_vit16_fc2": (16384, 1152, 4304),
    "mid_vit4_fc1": (4096, 4304, 1152), "mid_llm2k_o": (2048, 3584, 3584),
    "mid_llm2k_gu": (2048, 37888, 3584), "mid_llm1k_down": (1280, 3584, 18944),
    "vit64_qkv": (65536, 3456, 1152), "vit64_fc1": (65536, 4304, 1152), "sp8_gu": (8448, 37888, 3584),
}
out = ["# r02 — tcgen05 GEMM configurations vs cuBLAS on B200 (tools/bench_gemm.py, CUDA events, us per call,",
       "weights rotated through > L2 worth of copies)", "",
       "`dispatch` = what `vila_linear` picks by itself; the other columns force a kernel through `vila_linear_cfg`.", "",
       "| shape (M,N,K) | cuBLAS | " + " | ".join(names[c] for c in cfgs) + " |",
       "|---|---|" + "---|" * len(cfgs)]
for k, row in d.items():
    best = min((v for c, v in row.items() if c in cfgs and isinstance(v, (int, float))), default=None)
    cells = []
    for c in cfgs:
        v = row.get(c)
        if not isinstance(v, (int, float)):
            cells.append("-")
        else:
            cells.append(f"**{v}**" if v == best else f"{v}")
    out.append(f"| {k} {shapes.get(k, '')} | {row['cublas_us']} ({row['cublas_tflops']} TF) | " + " | ".join(cells) + " |")
out += ["", "Reading: CTA pairs (`tcgen05.mma.cta_group::2`, 256x256 tiles) win once they fill the SM pairs (large M);",
        "the swap-AB skinny kernel with cluster split-K wins for M = 279 (weights stream once); split-K CTA pairs",
        "(DSMEM exchange) win for long-K GEMMs with <= 74 tiles (ViT fc2); the single-CTA tiles cover the rest."]
Path("profiles/r02_gemm_configs.md").write_text("\n".join(out) + "\n")
print("\n".join(out))
