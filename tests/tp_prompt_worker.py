"""Worker of the tensor-parallel prompt check (launched by tests/test_gpu_tp.py through torch.distributed.run): 300 tokens on a sharded
model, so many that the last tiles of a rank's slice of W_down (512 x 2816 on two ranks) are shared between CTAs; logits against the whole model's, bit for bit."""
import os
import sys

import numpy as np

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))


def main():
    import torch
    import torch.distributed as dist
    from spy_b200 import backend as B
    from spy_b200 import gguf_io

    rank, world, local = int(os.environ["RANK"]), int(os.environ["WORLD_SIZE"]), int(os.environ["LOCAL_RANK"])
    os.environ.setdefault("NCCL_NVLS_ENABLE", "0")
    dist.init_process_group(backend="gloo", rank=rank, world_size=world)
    torch.cuda.set_device(local)
    cfg = gguf_io.LlamaConfig(n_layer=4, d_model=1024, n_head=8, n_ff=2816, n_vocab=2048, weight_std=0.03)
    if rank == 0:
        gguf_io.make_llama_gguf(sys.argv[1], cfg, seed=5)
    dist.barrier()
    be = B.B200Backend(local, tp_size=world, tp_rank=rank)
    m = B.LlamaModel(be, sys.argv[1], n_ctx=320)
    uid = [B.nccl_unique_id() if rank == 0 else None]
    dist.broadcast_object_list(uid, src=0)
    m.init_tp(uid[0])
    handles = [None] * world
    dist.all_gather_object(handles, m.tp_export())
    m.tp_import(handles)
    prompt = np.random.default_rng(6).integers(3, cfg.n_vocab, size=300)
    logits = m.eval(prompt, 0).copy()
    ok = True
    if rank == 0:
        b1 = B.B200Backend(local)
        m1 = B.LlamaModel(b1, sys.argv[1], n_ctx=320)
        ok = bool(np.array_equal(logits.view(np.uint32), m1.eval(prompt, 0).view(np.uint32)))
        print(f"TP{world} vs TP1: 300-token prompt bits identical = {ok} -> {'OK' if ok else 'FAIL'}", flush=True)
        m1.close(); b1.close()
    m.close(); be.close()
    flag = torch.tensor([0 if ok else 1])
    dist.all_reduce(flag)
    dist.destroy_process_group()
    sys.exit(int(flag.item() != 0))


if __name__ == "__main__":
    main()
