"""When the host pipeline issues, records and replays its schedule: the same on every rank, and only for the buffers recorded.
The schedule itself and the graph calls are stand-ins here (no GPU); the collectives run over gloo."""
import contextlib
import datetime
import os

import torch
import torch.distributed as dist
import torch.multiprocessing as mp

from megafold_b200 import host_pipeline


class Stream:
    def synchronize(self):
        pass

    def wait_stream(self, other):
        pass


class Graph:
    recording = None

    def __init__(self):
        self.steps = []

    def replay(self):
        for step in self.steps:
            step()


@contextlib.contextmanager
def record(graph, stream=None):
    Graph.recording = graph
    yield
    Graph.recording = None


class Pipeline(host_pipeline.HostPipeline):
    """Sums q over the ranks into d_bias; notes what it did."""

    def __init__(self):
        self.device, self.s_cap, self.out, self.did = torch.device("cpu"), Stream(), {}, []
        self.graph, self.graph_key, self.last_key, self.use_graph, self.group = None, None, None, True, None

    def _schedule(self, host, cur):
        def step(q=host["q"], group=self.group):
            d_bias = q.clone()
            if group is not None:
                dist.all_reduce(d_bias, group=group)
            self.out["d_bias"] = d_bias
        if Graph.recording is not None:
            self.did.append("record")
            Graph.recording.steps.append(step)
        else:
            self.did.append("issue")
            step()


def stand_in():
    torch.cuda.current_stream, torch.cuda.CUDAGraph, torch.cuda.graph = (lambda *a: Stream()), Graph, record
    torch.Tensor.is_pinned = lambda self: True


def _worker(rank, world, port, out):
    os.environ.update(MASTER_ADDR="127.0.0.1", MASTER_PORT=str(port))
    dist.init_process_group("gloo", rank=rank, world_size=world, timeout=datetime.timedelta(seconds=30))
    try:
        stand_in()
        group, pipe = dist.group.WORLD, Pipeline()
        rest = [torch.zeros(2) for _ in range(5)]
        fixed, turning = torch.zeros(3), [torch.zeros(3) for _ in range(2)]
        for step in range(8):
            # rank 0 comes with the same buffer every time; rank 1 alternates at first and then keeps one
            q = fixed if rank == 0 else turning[step % 2 if step < 4 else 0]
            q.fill_(10 * step + rank)
            pipe.run(q, *rest, group=group)
            assert torch.equal(pipe.out["d_bias"], torch.full((3,), 20.0 * step + 1)), (step, pipe.out)
        torch.save(pipe.did, os.path.join(out, f"r{rank}.pt"))
    finally:
        dist.destroy_process_group()


def test_ranks_take_the_same_steps(tmp_path):
    port = 33500 + os.getpid() % 2000
    mp.spawn(_worker, args=(2, port, str(tmp_path)), nprocs=2, join=True)
    did = [torch.load(os.path.join(tmp_path, f"r{r}.pt")) for r in range(2)]
    assert did[0] == did[1] == ["issue"] * 5 + ["record"]      # buffers of both ranks come back at the sixth call


def _one_process(_):
    stand_in()
    rest = [torch.zeros(2) for _ in range(5)]
    wide = torch.arange(12.0).view(4, 3)
    pipe = Pipeline()
    for _ in range(3):
        pipe.run(wide[:, :2], *rest)
    assert pipe.did == ["issue", "record"] and torch.equal(pipe.out["d_bias"], wide[:, :2])
    flat = torch.as_strided(wide, (4, 2), (2, 1))                 # the same address, other strides
    pipe.run(flat, *rest)
    assert pipe.did[2:] == ["issue"] and torch.equal(pipe.out["d_bias"], flat)


def test_graph_is_for_the_layout_it_recorded():
    mp.spawn(_one_process, nprocs=1, join=True)
