"""Mirror of the reference's ``src.serving`` package for the hot path (pipeline, cache manager,
real-model pipeline) and its HTTP front end (server.py)."""
