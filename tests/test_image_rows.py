"""A slab knows the rows of the whole image, the sum of all ranks' shares (gloo on the CPU)."""
import os
import socket

import torch
import torch.distributed as dist
import torch.multiprocessing as mp

from sapa_b200 import sharding


def _worker(rank, world, port, ret):
    os.environ["MASTER_ADDR"] = "127.0.0.1"
    os.environ["MASTER_PORT"] = str(port)
    dist.init_process_group("gloo", rank=rank, world_size=world)
    try:
        ret[rank] = sharding.RowSlab(1, 8, 16, 5 + rank, 16, torch.float32, torch.device("cpu")).image_rows
    finally:
        dist.destroy_process_group()


def test_image_rows():
    with socket.socket() as s:
        s.bind(("127.0.0.1", 0))
        port = s.getsockname()[1]
    with mp.Manager() as mgr:
        ret = mgr.dict()
        mp.spawn(_worker, args=(2, port, ret), nprocs=2, join=True)
        assert dict(ret) == {0: 11, 1: 11}
    assert sharding.RowSlab(1, 8, 16, 5, 16, torch.float32, torch.device("cpu")).image_rows == 0      # by itself: not known
