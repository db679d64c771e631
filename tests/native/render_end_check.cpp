// Host-side check of how a render's end is reported: each device error by its own status, the iteration
// limit only where there is none.
#include "pg_runtime.h"

#include <cstdio>
#include <cstring>

namespace
{

bool reported(uint32_t flags, bool done, int status, const char* text)
{
	try
	{
		pg::check_render_end(flags, done);
	}
	catch(const pg::Error& e)
	{
		const bool ok = e.status == status && std::strstr(e.what(), text);
		if(!ok)
		{
			std::printf("flags %u done %d: %d %s\n", flags, done ? 1 : 0, e.status, e.what());
		}
		return ok;
	}
	std::printf("flags %u done %d: no error\n", flags, done ? 1 : 0);
	return false;
}

}// end anonymous namespace

int main()
{
	pg::check_render_end(0u, true);
	if(!reported(pg::PG_DEV_ERR_STACK, true, pg::PG_ERR_STACK_OVERFLOW, "stack overflow") ||
	   !reported(pg::PG_DEV_ERR_STACK | pg::PG_DEV_ERR_QUEUE, false, pg::PG_ERR_STACK_OVERFLOW, "stack overflow") ||
	   !reported(pg::PG_DEV_ERR_QUEUE, false, pg::PG_ERR_QUEUE_OVERFLOW, "queues ran empty") ||
	   !reported(0u, false, pg::PG_ERR_ITERATION_LIMIT, "iteration limit"))
	{
		return 1;
	}
	std::puts("ok");
	return 0;
}
