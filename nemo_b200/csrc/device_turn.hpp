#ifndef NEMO_B200_DEVICE_TURN_HPP
#define NEMO_B200_DEVICE_TURN_HPP

/* The order of grids whose blocks wait for one another, on each device of the
 * process. Two such grids must not be partly resident at once: each would
 * hold SMs that the other's blocks need before its own can go on. There are
 * two kinds:
 *   - finite ones (the step kernel over several cycles, the one-launch LIF
 *     kernels): their launches are enclosed in a DeviceTurn, which makes the
 *     stream wait for the turn before (an event a device) and first ends a
 *     stay;
 *   - a stay: a step kernel that stays on the device and takes its commands
 *     from its host thread, for as long as that goes on calling. It starts
 *     with DeviceTurn::tryStay, when no finite grid is in flight, and ends at
 *     the next turn that another caller takes.
 * Kernels whose blocks wait for no other block need no turn.
 *
 * Any thread may take a turn. Locks are taken in one order: the device's
 * turn, then the stay's own (endStay). */

#include <atomic>

#include <cuda_runtime.h>

namespace nemo_b200 {

/* The owner of a stay */
class Stay {
public:
	/* End the launch and wait until it has left the device; nothing to do
	 * when it has already. From any thread, with the device's turn held. */
	virtual void endStay() noexcept = 0;
protected:
	~Stay() {}
};

struct TurnState;

class DeviceTurn {
public:
	/* The current device must be `device`, the stream one of its streams.
	 * self: a caller whose own stay, if any, is over already. */
	DeviceTurn(int device, cudaStream_t stream, const Stay* self = nullptr);
	~DeviceTurn();
	DeviceTurn(const DeviceTurn&) = delete;
	DeviceTurn& operator=(const DeviceTurn&) = delete;

	/* Start a stay: `launch` runs with the turn held, after another owner's
	 * stay has ended. False, with nothing done, while another thread has the
	 * turn or waits for it, or while a finite grid is in flight on another
	 * stream's behalf: the caller then goes without a stay (its launches must
	 * not wait for one another's blocks). */
	template<class Launch>
	static bool tryStay(int device, Stay* self, Launch launch)
	{
		TryLock turn(device, self);
		if(!turn.held) return false;
		launch();
		return true;
	}

	/* Another caller waits for the turn: a stay should end */
	static const std::atomic<int>* wanted(int device);

	/* The owner is about to be destroyed: afterwards nothing refers to it */
	static void leave(int device, const Stay* self);

private:
	struct TryLock {
		TryLock(int device, Stay* self);
		~TryLock();
		TurnState& s;
		bool held;
	};
	TurnState& m_s;
	cudaStream_t m_stream;
};

} // namespace nemo_b200

#endif
