#!/usr/bin/env python
"""Small single-GPU workloads for profiler captures (one kernel family per --case).

Each case launches its kernel a handful of times on inputs larger than the 126 MB L2 but well
under a few GB, so that `ncu --set full -k regex:<kernel> -c 1..3` finishes in a minute or two.
Multi-rank kernels run as emulated ranks (threads of this process, one cooperative grid).

    python bench/ncu_cases.py --case gemm
    ncu --set full --clock-control none -k regex:gemm_kernel -s 1 -c 1 -o /tmp/prof_gemm python bench/ncu_cases.py --case gemm
"""
import argparse
import os
import sys
import threading

import torch

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))


def emulated(world, fn):
    from asystem_amem_b200 import Communicator, get_unique_id
    uid = get_unique_id()
    errs = []

    def body(rank):
        try:
            torch.cuda.set_device(0)
            comm = Communicator(world, rank, uid)
            fn(rank, comm)
            torch.cuda.synchronize()
            comm.destroy()
        except BaseException as e:  # noqa: BLE001
            errs.append(repr(e))

    th = [threading.Thread(target=body, args=(r,)) for r in range(world)]
    [t.start() for t in th]
    [t.join() for t in th]
    if errs:
        raise SystemExit("; ".join(errs))


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--case", required=True)
    ap.add_argument("--reps", type=int, default=3)
    args = ap.parse_args()
    torch.cuda.set_device(0)
    reps = args.reps
    if args.case == "gemm":
        from asystem_amem_b200.ops import gemm_bf16
        a = torch.randn(8192, 8192, device="cuda").to(torch.bfloat16)
        b = (torch.randn(3584, 8192, device="cuda") * 0.02).to(torch.bfloat16)
        out = torch.empty(8192, 3584, device="cuda", dtype=torch.bfloat16)
        for _ in range(reps):
            gemm_bf16(a, b, out)
        torch.cuda.synchronize()
    elif args.case == "grouped_gemm":
        from asystem_amem_b200.ops import grouped_gemm_bf16, interleave_gate_up
        El, d, ffn, rows = 8, 4096, 1536, 32768
        counts = torch.tensor([5000, 3000, 4097, 4000, 1, 6670, 4000, 6000])
        offs = torch.zeros(El + 1, dtype=torch.int32)
        offs[1:] = counts.cumsum(0)
        offs = offs.cuda()
        x = torch.randn(rows, d, device="cuda").to(torch.bfloat16)
        w13 = interleave_gate_up((torch.randn(El, 2 * ffn, d, device="cuda") * 0.02).to(torch.bfloat16), ffn)
        act = torch.empty(rows, ffn, device="cuda", dtype=torch.bfloat16)
        for _ in range(reps):
            grouped_gemm_bf16(x, w13, offs, out=act, rows_hint=rows, swiglu=True)
        torch.cuda.synchronize()
    elif args.case == "one_gpu":
        # the kernels of the single-GPU paths in turn, inputs larger than L2 wherever the kernel is bound by memory
        from asystem_amem_b200 import Communicator, get_unique_id
        from asystem_amem_b200.models.llama import rope_tables
        from asystem_amem_b200.ops import MoeDispatcher, adamw_step, embedding, gemm_bf16, gemm_swiglu, rms_norm, rotate, route, swiglu
        from asystem_amem_b200.ops.elementwise import add_pieces
        from asystem_amem_b200.parallel.ep import ep_route_dispatch
        bf = lambda *s: torch.randn(*s, device="cuda").to(torch.bfloat16)  # noqa: E731
        comm = Communicator(1, 0, get_unique_id())
        x, w, w13, few = bf(2048, 8192), bf(4096, 8192), bf(2 * 8192, 8192), bf(16, 8192)
        src, wide = bf(100_000_000), torch.empty(100_000_000, device="cuda")
        dst = torch.empty_like(src)
        h, g = bf(4096, 2 * 14336).requires_grad_(True), bf(4096, 14336)
        f32 = [torch.rand(50_000_000, device="cuda") for _ in range(4)]
        T, E, k, d = 8192, 64, 8, 4096
        disp, tok = MoeDispatcher(comm, E, d, T * k), bf(T, d)
        top = torch.randn(T, E, device="cuda").topk(k, dim=1)
        idx, tw = top.indices.to(torch.int32), torch.softmax(top.values, dim=1)
        norm_x, norm_w = bf(32768, 4096).requires_grad_(True), bf(4096).requires_grad_(True)
        q, kk = bf(1, 8192, 32, 128).transpose(1, 2), bf(1, 8192, 8, 128).transpose(1, 2)
        rope = rope_tables(8192, 128, 500000.0, "cuda")
        table, ids = bf(65536, 4096).requires_grad_(True), torch.randint(0, 65536, (8192,), device="cuda")
        router, few_disp = bf(8, d).requires_grad_(True), MoeDispatcher(comm, 8, d, T * 2)
        tok_g = bf(T, d).requires_grad_(True)
        for _ in range(reps):
            torch.autograd.grad(rms_norm(norm_x, norm_w, 1e-5), (norm_x, norm_w), norm_x.detach())
            rotate(*rope, q, kk, as_they_lie=True)
            add_pieces(wide, [(0, src)])
            torch.autograd.grad(embedding(ids, table), table, tok)
            route(tok, router.detach(), 2)
            rows, _, _, _, top_w = ep_route_dispatch(few_disp, tok_g, router, 2)
            torch.autograd.grad([rows, top_w], (tok_g, router), [rows.detach(), top_w.detach()])
            gemm_bf16(x, w)
            gemm_bf16(few, w13[:7168])
            gemm_bf16(few, w13)
            gemm_swiglu(few, w13)
            comm.all_reduce(src, dst)
            comm.reduce_scatter(src, wide, scale=0.25)
            torch.autograd.grad(swiglu(h), h, g)
            adamw_step(*f32, src[:50_000_000], 1e-3, (0.9, 0.95), 1e-8, 0.0, 1)
            res = disp.dispatch(tok, idx)
            disp.combine(idx, tw, res.send_pos)
            disp.combine_grad_local(tok, disp.y, tw, res.send_pos)
        torch.cuda.synchronize()
        comm.destroy()
    elif args.case == "gradient_sums":
        # an embedding's gradient, tokens drawn evenly, half of them one id, and 70 an id; gradients into a shard, two sizes
        from asystem_amem_b200.ops import embedding
        from asystem_amem_b200.ops.elementwise import add_pieces
        table = torch.randn(32768, 4096, device="cuda").to(torch.bfloat16).requires_grad_(True)
        g, evenly = torch.randn(16384, 4096, device="cuda").to(torch.bfloat16), torch.randint(0, 32768, (16384,), device="cuda")
        half, often = torch.where(torch.rand(16384, device="cuda") < 0.5, 3, evenly), torch.arange(16384, device="cuda") % (16384 // 70)
        src, wide = torch.randn(100_000_000, device="cuda").to(torch.bfloat16), torch.zeros(100_000_000, device="cuda")
        for _ in range(reps):
            for ids in (evenly, half, often):
                torch.autograd.grad(embedding(ids, table), table, g)
            add_pieces(wide, [(0, src)])
        torch.cuda.synchronize()
    elif args.case == "window_allreduce":
        world = 4
        n = 32 << 20  # bf16 elements: 64 MiB per rank

        def fn(rank, comm):
            win = comm.window_alloc(n * 2)
            x = win.tensor(torch.bfloat16, n)
            x.normal_()
            torch.cuda.synchronize()
            for _ in range(reps):
                comm.all_reduce(x, algo="window")
            torch.cuda.synchronize()
            win.free()
        emulated(world, fn)
    elif args.case == "cublas":
        a = torch.randn(8192, 8192, device="cuda").to(torch.bfloat16)
        b = (torch.randn(3584, 8192, device="cuda") * 0.02).to(torch.bfloat16)
        out = torch.empty(8192, 3584, device="cuda", dtype=torch.bfloat16)
        for _ in range(reps):
            torch.matmul(a, b.t(), out=out)
        torch.cuda.synchronize()
    elif args.case in ("allreduce", "allgather", "reducescatter", "alltoall", "rs_cast"):
        world = 4
        n = 32 << 20  # bf16 elements per rank: 64 MiB per rank, 256 MiB over the emulated ranks

        def fn(rank, comm):
            x = torch.randn(n, device="cuda").to(torch.bfloat16)
            y = torch.empty(n, device="cuda", dtype=torch.bfloat16)
            for _ in range(reps):
                if args.case == "allreduce":
                    comm.all_reduce(x, y, algo="twoshot")
                elif args.case == "allgather":
                    comm.all_gather(x[: n // world], y)
                elif args.case == "reducescatter":
                    comm.reduce_scatter(x, y[: n // world])
                elif args.case == "rs_cast":
                    comm.reduce_scatter(x.float(), y[: n // world], scale=0.25)
                else:
                    comm.all_to_all(x, y)
        emulated(world, fn)
    elif args.case in ("ag_gemm", "gemm_rs"):
        from asystem_amem_b200.ops import all_gather_gemm, gemm_reduce_scatter
        world = 4

        def fn(rank, comm):
            if args.case == "ag_gemm":
                xs = torch.randn(1024, 8192, device="cuda").to(torch.bfloat16)
                w = (torch.randn(3584, 8192, device="cuda") * 0.02).to(torch.bfloat16)
                for _ in range(reps):
                    all_gather_gemm(comm, xs, w)
            else:
                h = torch.randn(4096, 3584, device="cuda").to(torch.bfloat16)
                w = (torch.randn(8192, 3584, device="cuda") * 0.02).to(torch.bfloat16)
                for _ in range(reps):
                    gemm_reduce_scatter(comm, h, w)
        emulated(world, fn)
    elif args.case == "moe":
        from asystem_amem_b200.ops import MoeDispatcher
        world, T, d, E, k = 4, 8192, 4096, 64, 8

        def fn(rank, comm):
            disp = MoeDispatcher(comm, E, d, 2 * T * k)
            x = torch.randn(T, d, device="cuda").to(torch.bfloat16)
            top = torch.randn(T, E, device="cuda").topk(k, dim=1)
            idx, w = top.indices.to(torch.int32), torch.softmax(top.values, dim=1)
            for _ in range(reps):
                res = disp.dispatch(x, idx)
                disp.combine(idx, w, res.send_pos)
        emulated(world, fn)
    else:
        raise SystemExit(f"unknown case {args.case}")
    print("done", args.case)


if __name__ == "__main__":
    main()
