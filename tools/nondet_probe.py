"""Repeat one W4A16 launch and describe how the results differ from the most common one (debugging aid)."""
import argparse, collections, os, sys
from pathlib import Path
import torch
sys.path.insert(0, str(Path(__file__).resolve().parent.parent))
import lite_llama_b200.kernels as K

ap = argparse.ArgumentParser()
ap.add_argument("--m", type=int, default=36); ap.add_argument("--n", type=int, default=4096); ap.add_argument("--k", type=int, default=14336)
ap.add_argument("--reps", type=int, default=200); ap.add_argument("--packed", type=int, default=1)
ap.add_argument("--const-zp", type=int, default=0); ap.add_argument("--const-sc", type=int, default=0); ap.add_argument("--const-x", type=int, default=0)
a = ap.parse_args()
torch.manual_seed(7)
x = torch.randn(a.m, a.k, device="cuda", dtype=torch.float16) * 0.5
qw = torch.randint(-(2**31), 2**31 - 1, (a.n, a.k // 8), device="cuda", dtype=torch.int64).to(torch.int32)
sc = torch.rand(a.n, a.k // 128, device="cuda") * 0.01 + 0.001
zp = torch.randint(0, 16, (a.n, a.k // 128), device="cuda").float()
if a.const_zp: zp.fill_(8.0)
if a.const_sc: sc.fill_(0.005)
if a.const_x: x.fill_(0.25)
pk = K.w4a16_pack(qw, sc, zp, group_size=128)
outs = []
for _ in range(a.reps):
    y = K.w4a16_matmul_packed(x, pk) if a.packed else K.w4a16_matmul(x, qw, sc, zp, group_size=128)
    torch.cuda.synchronize()
    outs.append(y.clone())
keys = collections.Counter(o.cpu().numpy().tobytes() for o in outs)
print(f"m={a.m} n={a.n} k={a.k} packed={a.packed} const zp/sc/x={a.const_zp}{a.const_sc}{a.const_x}: {len(keys)} distinct results in {a.reps} launches; counts {sorted(keys.values(), reverse=True)[:6]}")
ref = max(outs, key=lambda o: keys[o.cpu().numpy().tobytes()])
shown = 0
for i, o in enumerate(outs):
    d = (o.float() - ref.float()).abs()
    if d.max() > 0 and shown < 6:
        rows = torch.nonzero(d.amax(dim=1) > 0).flatten().tolist()
        cols = torch.nonzero(d.amax(dim=0) > 0).flatten().tolist()
        print(f"  launch {i}: {int((d > 0).sum())} elements differ, max abs {float(d.max()):.5f} (|y| max {float(ref.abs().max()):.2f}); token rows {rows[:12]}{'...' if len(rows) > 12 else ''} "
              f"cols {cols[0]}..{cols[-1]} ({len(cols)} cols; tiles {sorted(set(c // 128 for c in cols))[:10]})")
        shown += 1
