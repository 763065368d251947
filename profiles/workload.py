"""One pass through a part of the package at a small size, for a profiler: ``python profiles/workload.py pair|msa|recycle|layer_norm``."""
import os
import sys

import torch

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import protenix_b200 as px  # noqa: E402
from protenix_b200.init_utils import randomize_parameters_  # noqa: E402
from protenix_b200.msa import MSAModule  # noqa: E402


def main(part: str) -> None:
    torch.manual_seed(0)
    normal = lambda *shape: torch.randn(*shape, device="cuda")
    if part == "pair":              # one Pairformer block, fp32 z, with its single branch
        n = 768
        randomize_parameters_(px.PairformerBlock(), 1).cuda().eval()(normal(n, 384), normal(n, n, 128), None)
    elif part == "msa":             # two MSA blocks
        n, n_msa = 384, 1024
        mod = MSAModule(n_blocks=2, msa_configs={"strategy": "topk", "min_size": {"train": 1 << 20, "test": 1 << 20}})
        feat = {"msa": torch.randint(0, 32, (n_msa, n), device="cuda"), "has_deletion": torch.zeros(n_msa, n, device="cuda"),
                "deletion_value": torch.zeros(n_msa, n, device="cuda")}
        randomize_parameters_(mod, 1).cuda().eval()(feat, normal(n, n, 128), normal(n, 449), torch.ones(n, n, device="cuda"))
    elif part == "recycle":         # the pair update between two cycles
        n = 768
        trunk = randomize_parameters_(px.RecyclingTrunk(n_blocks=0), 1).cuda().eval()
        trunk.update_pair(normal(n, n, 128), normal(n, n, 128))
    elif part == "layer_norm":      # the op, forward and backward, on a pair tensor in bf16
        ln = randomize_parameters_(px.LayerNorm(128), 1).cuda()
        x = normal(768 * 768, 128).bfloat16().requires_grad_()
        ln(x).backward(torch.ones_like(x))
    else:
        raise SystemExit(__doc__)
    torch.cuda.synchronize()


if __name__ == "__main__":
    main(sys.argv[1] if len(sys.argv) > 1 else "")
