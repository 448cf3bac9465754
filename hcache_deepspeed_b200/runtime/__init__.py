"""Training runtime (``deepspeed.initialize`` side of the reference: ``deepspeed/runtime``). It is
kept functional and torch.distributed-native (NCCL on GPUs, gloo in CPU tests) rather than kernel-optimised."""
